// CRS_MODE_FP64: wdot by tiles of 32 states in 64-bit fixed point and FP64.
//
// What bounds it.  The FP64 pipe retires one warp instruction per SM sub-
// partition in ~70 clocks, so 15,000 FP64 instructions per state (53
// species / 325 reactions) held the one-state-per-thread kernel at 33.6 M
// states/s, 95% of that pipe.  Of the arithmetic here only the sums keep
// FP64: the mass-fraction sums in the reference's order and one
// multiply-add per nonzero net stoichiometric coefficient.  Everything
// multiplicative -- rate constants, equilibrium constants, concentrations,
// third bodies, fall-off -- is an exponent in 64-bit fixed point
// (crs_fx.cuh): a product of factors is a sum of integers, a rate constant
// a dot product of a reaction's coefficients with functions of T that are
// formed once per state, and each rate one table exponential.
//
// A reaction's exponents.  On a temperature interval (bounded by the
// mechanism's T_common values and the limits TLO, THI) with centre and
// half width of log2 T, 1/T and T, the functions L, I, t, t^2, t^3, t^4 are
// normalised to [-1, 1] and every exponent is c0 + cL L + cI I + c1 t + ...
// + c4 t^4: three coefficients forward; the reverse rate's exponent, forward
// minus ln Kc with the Gibbs polynomials of all its species, has seven.
// Coefficients are rounded to 2^-52, the functions to 2^-61.
//
// A tile: lane = state; the CTA's NW warps share the tile's exponents of
// the concentrations ([N][32], 8 bytes each) and split first the species,
// then the reactions (lists balanced at load by instruction counts), then
// the species sums.  The net rates pass between the last two in shared
// memory ([R][32]) or, when they do not fit, in global scratch of one tile
// per CTA, which stays in L2.  Table reads are uniform across a warp up to
// the temperature interval and go through L1.
//
// States outside the scheme (T outside (TLO, THI], a non-positive or non-
// finite density, |Y| >= 2, a subnormal Y) and reactions outside it (non-
// integer coefficients, PLOG, Chebyshev, coefficients beyond the bounds)
// are evaluated lane by lane by the general FP64 arithmetic (slow_net).
#include <cuda_runtime.h>
#include <math.h>

#include "crs_fast.cuh"
#include "crs_fx.cuh"
#include "crs_fx_tab.cuh"
#include "crs_internal.cuh"
#include "crs_tile.cuh"

namespace crs {
namespace fx {

constexpr int64_t ZMIN = -561023779885736503LL;   // log2 1e-300
constexpr int64_t LOG2_10 = 1870079266285788LL;   // log2 10
constexpr int64_t C04 = 748031706514315LL;        // 0.4 log2 10
constexpr int64_t C0806 = 1507283888626345LL;     // 0.806 log2 10
constexpr int64_t K067 = 3089829632346349896LL;   // 0.67, 2^-62
constexpr int64_t K11762 = 5424265094874293653LL; // 1.1762
constexpr int64_t K014 = 645636042579834307LL;    // 0.14

// The lane's functions of T.
struct Basis {
  Dg L, I, t1, t2, t3, t4;
};
// rows of the per-tile block: the six functions, log2 rho, the mean 1/W,
// y_N, rho, and the interval and the outside-the-scheme mark
constexpr int ROWS = 11;

__device__ __forceinline__ Dg dg(int2 v) { return Dg{v.x, v.y}; }
__device__ __forceinline__ int64_t word(int hi, int lo) {
  return (int64_t)(((uint64_t)(unsigned)hi << 32) | (unsigned)lo);
}
__device__ __forceinline__ int64_t word(int2 v) { return word(v.x, v.y); }

struct Dot {
  int64_t hh, mid;
  __device__ __forceinline__ explicit Dot(int64_t c0) : hh(c0), mid(1LL << 31) {}
  __device__ __forceinline__ void add(Dg c, Dg f) {
    hh = mad(c.hi, f.hi, hh);
    mid = mad(c.lo, f.hi, mad(c.hi, f.lo, mid));
  }
  __device__ __forceinline__ int64_t exponent() const { return even(hh + (mid >> 32)); }
};

// log2 of a fall-off factor from lth = log2 [M] (c: its record on the lane's
// interval).  slow: outside the scheme (negative or tiny terms); the caller
// evaluates the reaction in FP64.
__device__ __noinline__ int64_t falloff(const int2 *__restrict__ c, int flags, int64_t lth,
                                        Dg L, Dg I, Dg t, const int64_t *et, const int64_t *lt,
                                        bool &slow) {
  Dot d(word(c[0]));
  d.add(dg(c[1]), L);
  d.add(dg(c[2]), I);
  const int64_t z = d.exponent() + lth;  // log2 Pr
  slow |= z & 1;
  // log2(1 + Pr) = max(z, 0) + log2(1 + 2^-|z|)
  uint64_t M;
  int E;
  exp2m(z < 0 ? z : -z, et, M, E);
  int64_t w = (int64_t)((M << 6) >> min(-E, 63));
  if (w >> 62) w = (1LL << 62) - 1;
  const int64_t lv = log2m((uint64_t)((1LL << 62) + w) << 1, lt);
  int64_t f = ((flags & PMF_LOW) ? (z < 0 ? z : 0) : (z > 0 ? -z : 0)) - lv;
  if (!(flags & (PMF_TROE | PMF_SRI))) return even(f);
  const int64_t zP = z > ZMIN ? z : ZMIN;
  // Fcent (Troe) or the base of the SRI power, in units of 2^-59
  int64_t S = 0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (flags & (PMF_T1 << q)) {
      const int64_t y = word(c[3 + 2 * q]);
      exp2m(y + mul<0>(dg(c[4 + 2 * q]), q == 2 ? I : t), et, M, E);
      slow |= E > 1;
      const int64_t v = (int64_t)((M << 6) >> min(max(3 - E, 2), 63));
      S += (y & 1) ? -v : v;
    }
  }
  slow |= S < (1LL << 39);
  const int64_t zF = log2i(S > 1 ? S : 1, 59, lt);
  int64_t A = zP, B = LOG2_10;
  if (flags & PMF_TROE) {
    const Dg kF = split(zF);
    A = zP - mul<2>(kF, split(K067)) - C04;
    B = C0806 - mul<2>(kF, split(K11762)) - mul<2>(split(zP), split(K014));
  }
  bool ok;
  const int64_t rho = ratio2(A, B, ok);
  slow |= !ok;
  f += mul<3>(split(zF), split(rho));
  if (flags & PMF_DE) {
    Dot e(word(c[9]));
    e.add(dg(c[10]), L);
    f += e.exponent();
  }
  return even(f);
}

// Concentrations of one state from its mass fractions (slow_net).
struct YConc {
  const double *Y;
  int64_t ld;
  double rho, yN;
  const double *inv_mw;
  int N;
  __device__ double operator[](int k) const {
    return (k == N - 1 ? yN : Y[(int64_t)k * ld]) * (rho * inv_mw[k]);
  }
};

// The net rate of reaction r by the general FP64 arithmetic.
__device__ __noinline__ double slow_net(const unsigned char *img, const ImgLayout &lay, int r,
                                        double T, double P, const double *Y, int64_t ld,
                                        double rho, double yN) {
  const Tab t = make_tab(img, lay);
  fast::State s;
  s.T = T;
  s.P = P;
  s.invT = 1.0 / T;
  s.logT = fast::log_t(T, t.logtab);
  s.tab = t.exptab;
  s.ltab = t.logtab;
  KcPolyG kc;
  kc.T = T;
  kc.logT = s.logT;
  kc.invT = s.invT;
  double fwd, rev, pm;
  return fast::rxn_net(t, r, s, P * s.invT * fast::INV_RU, YConc{Y, ld, rho, yN, t.inv_mw, t.N},
                       kc, fwd, rev, pm);
}

template <bool REV>
__device__ __noinline__ double net_far(int64_t yf, int64_t yr, const int64_t *tab) {
  return net_special<REV>(yf, yr, tab);
}

// The normalised functions of T of one state into column `lane` of the
// block; returns the temperature interval.  irr: T outside the scheme.
__device__ __forceinline__ int basis_of(const FxTab &f, const unsigned char *tab, double T,
                                        int64_t *blk, bool &irr) {
  irr = !(T > f.tb[0] && T <= f.tb[NI]);
  const double Tc = irr ? 1000.0 : T;
  int iv = 0;
#pragma unroll
  for (int q = 1; q < NI; ++q) iv += Tc > f.tb[q];
  const int64_t *w = reinterpret_cast<const int64_t *>(tab + f.basis) + BASIS * iv;
  const int64_t *hp = reinterpret_cast<const int64_t *>(tab + f.hp);
  const Dg L = split(mul<2>(split((log2hp(Tc, hp) - w[3]) << w[5]), split(w[4])));
  const Dg t = split(mul<2>(split((d2fx(Tc, 49) - w[0]) << w[2]), split(w[1])));
  // 1/T to 2^-68: the rounded reciprocal and its residual
  const double r = 1.0 / Tc, e = fma(-Tc, r, 1.0) * r;
  const int64_t x = d2fx(r, 68) + (int64_t)(float)(e * 0x1p68);
  const Dg I = split(mul<2>(split((x - w[6]) << w[8]), split(w[7])));
  // powers: 2^-61 2^-61 -> 2^-61
  const Dg t2 = split(mul<3>(t, t));
  const Dg t3 = split(mul<3>(t2, t)), t4 = split(mul<3>(t2, t2));
  int2 *o = reinterpret_cast<int2 *>(blk);
  o[0] = make_int2(L.hi, L.lo);
  o[32] = make_int2(I.hi, I.lo);
  o[64] = make_int2(t.hi, t.lo);
  o[96] = make_int2(t2.hi, t2.lo);
  o[128] = make_int2(t3.hi, t3.lo);
  o[160] = make_int2(t4.hi, t4.lo);
  return iv;
}

struct Args {
  const unsigned char *img;  // table image (general FP64 arithmetic, sums)
  const unsigned char *tab;  // fixed-point tables
  double *q;                 // [gridDim.x][R][32] scratch when QS is false
};

// U plain reversible reactions at once: exponents, rates, net rates into q.
template <int U>
__device__ __forceinline__ void plain_block(const FxTab &f, const unsigned char *tab,
                                            const int *list, const int64_t *yl, const Basis &B,
                                            int iv, double T, const int64_t *et,
                                            double *q) {
  int64_t yf[U], yr[U];
  int r[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    r[u] = list[u];
    const int4 h0 = __ldg(reinterpret_cast<const int4 *>(tab + f.hdr) + 2 * r[u]);
    const int4 h1 = __ldg(reinterpret_cast<const int4 *>(tab + f.hdr) + 2 * r[u] + 1);
    int idx = iv;
    if (!f.uniform) {
      const int32_t *tp = reinterpret_cast<const int32_t *>(tab + f.thr_ptr);
      idx = 0;
      for (int e = tp[r[u]]; e < tp[r[u] + 1]; ++e)
        idx += T > reinterpret_cast<const double *>(tab + f.thr)[e];
    }
    const int4 *c = reinterpret_cast<const int4 *>(tab + f.coef) + 5 * (h0.z + idx);
    const int4 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2), c3 = __ldg(c + 3),
               c4 = __ldg(c + 4);
    Dot a(word(c0.x, c0.y));
    a.add(Dg{c0.z, c0.w}, B.L);
    a.add(Dg{c1.x, c1.y}, B.I);
    Dot b(word(c1.z, c1.w));
    b.add(Dg{c2.x, c2.y}, B.L);
    b.add(Dg{c2.z, c2.w}, B.I);
    b.add(Dg{c3.x, c3.y}, B.t1);
    b.add(Dg{c3.z, c3.w}, B.t2);
    b.add(Dg{c4.x, c4.y}, B.t3);
    b.add(Dg{c4.z, c4.w}, B.t4);
    const int neg = (h0.y & RF_NEG) ? 1 : 0;
    int64_t sf = yl[(h1.x & 0xffff) * 32] + yl[((unsigned)h1.x >> 16) * 32];
    int64_t sr = yl[(h1.z & 0xffff) * 32] + yl[((unsigned)h1.z >> 16) * 32];
    if (h0.y & RF_MORE_R) sf += yl[(h1.y & 0xffff) * 32] + yl[((unsigned)h1.y >> 16) * 32];
    if (h0.y & RF_MORE_P) sr += yl[(h1.w & 0xffff) * 32] + yl[((unsigned)h1.w >> 16) * 32];
    yf[u] = a.exponent() + neg + sf;
    yr[u] = b.exponent() + neg + sr;
  }
  double v[U];
  bool sp[U], any = false;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    v[u] = net_of<true>(yf[u], yr[u], et, sp[u]);
    any |= sp[u];
  }
  if (any) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (sp[u]) v[u] = net_far<true>(yf[u], yr[u], et);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) q[(int64_t)r[u] * 32] = v[u];
}

template <int LIST, bool QS, bool TS>
__global__ void __launch_bounds__(warps_of(LIST) * 32, 16 / warps_of(LIST))
    k_wdot_tile(const __grid_constant__ ImgLayout lay, const __grid_constant__ FxTab f, Args g,
                Batch b) {
  constexpr int NW = warps_of(LIST);
  extern __shared__ __align__(128) unsigned char smem[];
  const int N = f.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned char *tab = g.tab;
  int64_t *yl = reinterpret_cast<int64_t *>(smem) + lane;         // [N + 1][32]
  int64_t *blk = yl + (N + 1) * 32;                               // [ROWS][32]
  double *s_yN = reinterpret_cast<double *>(blk + 8 * 32 - lane), *s_rho = s_yN + 32;
  int *s_iv = reinterpret_cast<int *>(s_yN + 64), *s_irr = s_iv + 32;
  int64_t *next = reinterpret_cast<int64_t *>(smem) + (N + 1 + ROWS) * 32;
  const int64_t *et = reinterpret_cast<const int64_t *>(tab + f.small);
  if (TS) {
    for (int k = threadIdx.x; k < TAB_BYTES / 8; k += NW * 32) next[k] = et[k];
    et = next;
    next += TAB_BYTES / 8;
  }
  const int64_t *lt = et + EXP_ENTRIES;
  double *q = (QS ? reinterpret_cast<double *>(next)
                  : g.q + (int64_t)blockIdx.x * f.R * 32) + lane;
  if (warp == 0) yl[N * 32] = 0;
  const Tab t = make_tab(g.img, lay);
  const double *inv_mw = t.inv_mw;
  const int64_t *lw = reinterpret_cast<const int64_t *>(tab + f.lw);
  const int *list = reinterpret_cast<const int *>(tab + f.list[LIST]);
  const int l0 = reinterpret_cast<const int *>(tab + f.list_ptr[LIST])[warp];
  const int l1 = reinterpret_cast<const int *>(tab + f.list_ptr[LIST])[warp + 1];
  const int lr = l0 + reinterpret_cast<const int *>(tab + f.list_rev[LIST])[warp];
  const int *sum = reinterpret_cast<const int *>(tab + f.sum[LIST]);
  const int s0 = reinterpret_cast<const int *>(tab + f.sum_ptr[LIST])[warp];
  const int s1 = reinterpret_cast<const int *>(tab + f.sum_ptr[LIST])[warp + 1];
  int bad = 0;
  for (int64_t tile = blockIdx.x; tile * 32 < b.n; tile += gridDim.x) {
    const int64_t i = tile * 32 + lane;
    const bool valid = i < b.n;
    const int64_t ic = valid ? i : tile * 32;  // idle lanes repeat a valid state
    const double T = b.T[ic], P = b.P[ic];
    // mass fractions on chip; the last warp also forms the functions of T
#pragma unroll 4
    for (int k = warp; k < N - 1; k += NW)
      yl[k * 32] = __double_as_longlong(b.Y[(int64_t)k * b.ld + ic]);
    if (warp == NW - 1) {
      bool irr;
      s_iv[lane] = basis_of(f, tab, T, blk, irr);
      s_irr[lane] = irr;
    }
    __syncthreads();
    // y_N = 1 - sum y in the reference's order (rate_subs.py:1312-1320) on
    // warp 0, the density on warp 1: two dependent FP64 chains side by side
    if (warp == 0) {
      double ys = N > 1 ? __longlong_as_double(yl[0]) : 0.0;
      for (int k = 1; k < N - 1; ++k) ys += __longlong_as_double(yl[k * 32]);
      s_yN[lane] = 1.0 - ys;
      yl[(N - 1) * 32] = __double_as_longlong(1.0 - ys);
      asm volatile("bar.sync 1, 64;" ::: "memory");
    } else if (warp == 1) {
      double mwi = 0.0;
      for (int k = 0; k < N - 1; ++k) mwi = fma(__longlong_as_double(yl[k * 32]), inv_mw[k], mwi);
      asm volatile("bar.sync 1, 64;" ::: "memory");
      mwi = fma(s_yN[lane], inv_mw[N - 1], mwi);
      const double rho = P / mwi * ((1.0 / T) * fast::INV_RU);
      s_rho[lane] = rho;
      // a positive density of moderate size, a mean 1/W below 2
      const int e = (int)(bits_of(rho) >> 52), m = (int)(bits_of(mwi) >> 52);
      if (e < 1023 - 400 || e > 1023 + 400 || m < 1023 - 40 || m > 1023) s_irr[lane] = 1;
      blk[6 * 32] = even(log2d(rho, lt));
      blk[7 * 32] = d2fx(mwi, 61 - f.eff_shift);
    }
    __syncthreads();
    const int64_t lrho = blk[6 * 32];
    // third-body concentrations: [M] = rho (1/mw + sum (eff - 1) Y / W), as
    // exponents into the slots of their reactions' rates
    if (f.NPM > 0) {
      const int4 *pmh = reinterpret_cast<const int4 *>(tab + f.pmh);
      const int *ep = reinterpret_cast<const int *>(tab + f.eff_ptr);
      const int *es = reinterpret_cast<const int *>(tab + f.eff_sp);
      const int2 *ek = reinterpret_cast<const int2 *>(tab + f.eff_k);
      const int64_t m = blk[7 * 32];
      for (int p = warp; p < f.NPM; p += NW) {
        const int4 h = __ldg(pmh + p);
        if (!(h.x & PMF_SUM)) continue;
        int64_t s = m;
        for (int e = ep[p]; e < ep[p + 1]; ++e)
          s += mul<4>(dg(__ldg(ek + e)), split(d2fx(__longlong_as_double(yl[es[e] * 32]), 60)));
        const int64_t a = s < 0 ? -s : s;
        int64_t l = even(log2i(a | (a == 0), 61 - f.eff_shift, lt) + lrho) | (s < 0);
        if (a == 0) l = ZERO_EXP;
        q[(int64_t)h.z * 32] = __longlong_as_double(l);
      }
      __syncthreads();
    }
    // exponents of the concentrations in place of the mass fractions
    for (int k = warp; k < N; k += NW) {
      const double y = __longlong_as_double(yl[k * 32]);
      const uint64_t u = bits_of(y);
      const int e = (int)(u >> 52) & 0x7ff;
      int64_t l = even(log2d(y, lt) + lw[k] + lrho) | (int64_t)(u >> 63);
      if ((u << 1) == 0) l = ZERO_EXP;
      else if (e == 0 || e > 1023) s_irr[lane] = 1;  // subnormal, |y| >= 2, NaN
      yl[k * 32] = l;
    }
    __syncthreads();
    // net rates
    const bool irr = s_irr[lane] != 0;
    {
      const int iv = s_iv[lane];
      Basis B;
      const int2 *o = reinterpret_cast<const int2 *>(blk);
      B.L = dg(o[0]);
      B.I = dg(o[32]);
      B.t1 = dg(o[64]);
      B.t2 = dg(o[96]);
      B.t3 = dg(o[128]);
      B.t4 = dg(o[160]);
      int p = l0;
      for (; p + 2 <= lr; p += 2) plain_block<2>(f, tab, list + p, yl, B, iv, T, et, q);
      for (; p < lr; ++p) plain_block<1>(f, tab, list + p, yl, B, iv, T, et, q);
      for (; p < l1; ++p) {
        const int r = list[p];
        const int4 h0 = __ldg(reinterpret_cast<const int4 *>(tab + f.hdr) + 2 * r);
        const int4 h1 = __ldg(reinterpret_cast<const int4 *>(tab + f.hdr) + 2 * r + 1);
        bool slow = (h0.y & RF_GEN) != 0;
        double v = 0.0;
        if (!(h0.y & RF_GEN)) {
          int idx = iv;
          if (!f.uniform) {
            const int32_t *tp = reinterpret_cast<const int32_t *>(tab + f.thr_ptr);
            idx = 0;
            for (int e = tp[r]; e < tp[r + 1]; ++e)
              idx += T > reinterpret_cast<const double *>(tab + f.thr)[e];
          }
          const int2 *c = reinterpret_cast<const int2 *>(tab + f.coef) + COEF * (h0.z + idx);
          int64_t l = (h0.y & RF_NEG) ? 1 : 0;  // what both directions share
          if (h0.w >= 0) {
            const int4 ph = __ldg(reinterpret_cast<const int4 *>(tab + f.pmh) + h0.w);
            int64_t lth = ph.y >= 0 ? yl[ph.y * 32]
                                    : __double_as_longlong(q[(int64_t)r * 32]);
            if (h0.y & RF_FALL)
              lth = falloff(reinterpret_cast<const int2 *>(tab + f.pmc) + PMC * (NI * h0.w + iv),
                            ph.x, lth, B.L, B.I, B.t1, et, lt, slow);
            l += lth;
          }
          Dot a(word(c[0]));
          a.add(dg(c[1]), B.L);
          a.add(dg(c[2]), B.I);
          int64_t yf = a.exponent() + l + yl[(h1.x & 0xffff) * 32] +
                       yl[((unsigned)h1.x >> 16) * 32];
          if (h0.y & RF_MORE_R)
            yf += yl[(h1.y & 0xffff) * 32] + yl[((unsigned)h1.y >> 16) * 32];
          bool sp;
          if (h0.y & RF_REV) {
            Dot d(word(c[3]));
            d.add(dg(c[4]), B.L);
            d.add(dg(c[5]), B.I);
            d.add(dg(c[6]), B.t1);
            d.add(dg(c[7]), B.t2);
            d.add(dg(c[8]), B.t3);
            d.add(dg(c[9]), B.t4);
            int64_t yr = d.exponent() + l + yl[(h1.z & 0xffff) * 32] +
                         yl[((unsigned)h1.z >> 16) * 32];
            if (h0.y & RF_MORE_P)
              yr += yl[(h1.w & 0xffff) * 32] + yl[((unsigned)h1.w >> 16) * 32];
            v = net_of<true>(yf, yr, et, sp);
            if (sp) v = net_far<true>(yf, yr, et);
          } else {
            v = net_of<false>(yf, 0, et, sp);
            if (sp) v = net_far<false>(yf, 0, et);
          }
        }
        if (slow)
          v = slow_net(g.img, lay, r, T, P, b.Y + ic, b.ld, s_rho[lane], s_yN[lane]);
        q[(int64_t)r * 32] = v;
      }
      if (irr)  // the state is outside the scheme: every rate in FP64
        for (p = l0; p < l1; ++p)
          q[(int64_t)list[p] * 32] =
              slow_net(g.img, lay, list[p], T, P, b.Y + ic, b.ld, s_rho[lane], s_yN[lane]);
    }
    __syncthreads();
    // species sums
    for (int a = s0; a < s1; ++a) {
      const int k = sum[a];
      const int e1 = t.spc_ptr[k + 1];
      int e = t.spc_ptr[k];
      double w = 0.0, w2 = 0.0;
      for (; e + 4 <= e1; e += 4) {
        double v[4], nu[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          v[u] = q[(int64_t)t.spc_r[e + u] * 32];
          nu[u] = t.spc_nu[e + u];
        }
        w = fma(nu[0], v[0], w);
        w2 = fma(nu[1], v[1], w2);
        w = fma(nu[2], v[2], w);
        w2 = fma(nu[3], v[3], w2);
      }
      for (; e < e1; ++e) w = fma(t.spc_nu[e], q[(int64_t)t.spc_r[e] * 32], w);
      w += w2;
      if (valid) {
        bad += ((__double2hiint(w) >> 20) & 0x7ff) == 0x7ff;  // inf or NaN, integer test
        b.wdot[(int64_t)k * b.ld + i] = w;
      }
    }
    // the next tile's mass fractions replace exponents that every warp is
    // done with (the barrier before the sums); its third bodies replace
    // rates only after two more barriers
  }
  if (bad && b.status) atomicAdd(&b.status[1], bad);
}

size_t smem_of(const FxTab &f, bool qs, bool ts) {
  return (size_t)(f.N + 1 + ROWS) * 256 + (ts ? TAB_BYTES : 0) + (qs ? (size_t)f.R * 256 : 0);
}

}  // namespace fx

// Scratch bytes of a launch over n states (0: the net rates fit on chip);
// < 0: the mechanism does not fit this kernel.
long long fx_scratch(const fx::FxTab &f, int64_t n, int sm_count, int smem_optin) {
  if (!f.usable) return -1;
  if (fx::smem_of(f, true, true) <= (size_t)smem_optin) return 0;
  if (fx::smem_of(f, false, false) > (size_t)smem_optin) return -1;
  const int64_t tiles = (n + 31) / 32;
  return (long long)(tiles < sm_count ? tiles : sm_count) * f.R * 256;
}

cudaError_t launch_wdot_fx(const unsigned char *img, const ImgLayout &L, const fx::FxTab &f,
                           const unsigned char *tab, const Batch &b, int sm_count,
                           int smem_optin, double *scratch, cudaStream_t s) {
  using fx::k_wdot_tile;
  const fx::Args g{img, tab, scratch};
  const int64_t tiles = (b.n + 31) / 32;
  const bool qs = !scratch;
  const bool ts = fx::smem_of(f, qs, true) <= (size_t)smem_optin;
  // sixteen warps per SM: in one CTA where tiles are few or large
  int list = 2;
  if (qs) {
    const size_t need = fx::smem_of(f, true, true) + 2048;
    if (4 * need <= (size_t)smem_optin && f.R < 100) list = 0;
    else if (2 * need <= (size_t)smem_optin) list = 1;
    if (list == 1 && tiles <= sm_count) list = 2;
  }
  const int per_sm = 16 / fx::warps_of(list);
  const size_t bytes = fx::smem_of(f, qs, ts);
  void (*k)(const ImgLayout, const fx::FxTab, fx::Args, Batch);
  if (qs) k = list == 0 ? k_wdot_tile<0, true, true> : list == 1 ? k_wdot_tile<1, true, true>
                                                                 : k_wdot_tile<2, true, true>;
  else k = ts ? k_wdot_tile<2, false, true> : k_wdot_tile<2, false, false>;
  const cudaError_t e = set_smem_limit(k, bytes);
  if (e != cudaSuccess) return e;
  const int64_t cap = (int64_t)sm_count * per_sm;
  k<<<(unsigned)(tiles < cap ? tiles : cap), fx::warps_of(list) * 32, bytes, s>>>(L, f, g, b);
  return cudaGetLastError();
}

}  // namespace crs
