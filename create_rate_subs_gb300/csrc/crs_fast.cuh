// General FP64 arithmetic of one reaction for one state: any rate form,
// pressure modification, non-integer coefficients.  Shared by the one-
// state-per-thread and warp kernels (crs_fast.cu) and, for the states and
// reactions its fixed-point scheme leaves out, by the state-tile kernel
// (crs_fx.cu).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "crs_exp.cuh"
#include "crs_internal.cuh"

namespace crs {
namespace fast {

using texp::exp_core;
using texp::exp_fix;
using texp::exp_t;
using texp::log_t;
constexpr double INV_RU = 0.0001202723625380408;
constexpr double LN10 = 2.302585092994046;
constexpr double INV_LN10 = 0.4342944819032518;

struct Col {
  double *p;
  int64_t stride;
  __device__ double &operator[](int k) const { return p[(int64_t)k * stride]; }
};

// Contiguous per-warp array (warp-per-state kernels).
struct Arr {
  double *p;
  __device__ double &operator[](int k) const { return p[k]; }
};

// Kc exponent from the per-species Gibbs column S: ln(prefactor) +
// sum_k nu_k S_k (the layouts that keep S on chip).
template <class CS>
struct KcCol {
  CS S;
  __device__ __forceinline__ double operator()(const Tab &t, int r, int j) const {
    double g = t.kc_lpref[j];
    for (int e = t.nu_ptr[r]; e < t.nu_ptr[r + 1]; ++e) g = fma(t.nu_val[e], S[t.nu_sp[e]], g);
    return g;
  }
};
template <class T>
struct IsKcCol { static constexpr bool value = false; };
template <class CS>
struct IsKcCol<KcCol<CS>> { static constexpr bool value = true; };

struct State {
  double T, invT, logT, P;
  const double *tab;   // 2^(j/256), exp_t
  const double *ltab;  // (1/F, log F), log_t
};

// Rate constant of row `row`; *x receives its exponent for the EXP kind.
__device__ __forceinline__ double rate(const Tab &t, int row, const State &s,
                                       double &x) {
  const double *c = t.rate_x + 3 * row;  // (logA | A), b, -Ta
  switch (t.rate_kind[row]) {
    case RATE_EXP:
      x = fma(c[2], s.invT, fma(c[1], s.logT, c[0]));
      return exp_t(x, s.tab);
    case RATE_CONST:
      return c[0];
    case RATE_NEGEXP:
      return c[0] * exp_t(fma(c[2], s.invT, c[1] * s.logT), s.tab);
    case RATE_POW: {
      double k = c[0];
      for (int j = 0; j < t.rate_npow[row]; ++j) k *= s.T;
      return k;
    }
    default:  // PLOG, Chebyshev
      return pdep_kf(t, row, s.T, s.logT, s.P);
  }
}

template <class CS>
__device__ __forceinline__ double product(const int32_t *sp, const int32_t *nint,
                                          const double *nu, int a, int b,
                                          const CS &C) {
  double p = 1.0;
  for (int j = a; j < b; ++j) {
    const double c = C[sp[j]];
    const int n = nint[j];
    if (n == 1) p *= c;
    else if (n == 2) p *= c * c;
    else if (n >= 0) for (int q = 0; q < n; ++q) p *= c;
    else p *= pow(c, nu[j]);
  }
  return p;
}

template <class CS>
__device__ double pres_mod(const Tab &t, int p, const State &s, double mix,
                           const CS &C) {
  double thd = mix;
  const int sp = t.pm_sp[p];
  if (t.pm_kind[p] == PM_THD || sp < 0) {
    for (int e = t.pm_eff_ptr[p]; e < t.pm_eff_ptr[p + 1]; ++e)
      thd = fma(t.pm_eff_val[e], C[t.pm_eff_sp[e]], thd);
    if (t.pm_kind[p] == PM_THD) return thd;
  } else {
    thd = C[sp];
  }
  const int r0 = t.pm_k0[p], ri = t.pm_kinf[p];
  double Pr;
  if (t.rate_kind[r0] == RATE_EXP && t.rate_kind[ri] == RATE_EXP) {
    const double *a = t.rate_x + 3 * r0, *b = t.rate_x + 3 * ri;
    const double x0 = fma(a[2], s.invT, fma(a[1], s.logT, a[0]));
    const double xi = fma(b[2], s.invT, fma(b[1], s.logT, b[0]));
    Pr = exp_t(x0 - xi, s.tab) * thd;
  } else {
    double x;
    const double k0 = rate(t, r0, s, x);
    const double ki = rate(t, ri, s, x);
    Pr = k0 * thd / ki;
  }
  const bool low = t.pm_kind[p] == PM_FALL_LOW;
  const double inv1p = 1.0 / (1.0 + Pr);
  const int form = t.pm_form[p];
  if (form == FORM_LINDEMANN) return low ? Pr * inv1p : inv1p;
  const double lP = log_t(fmax(Pr, 1.0e-300), s.ltab) * INV_LN10;
  double F;
  if (form == FORM_TROE) {
    const double *c = t.troe_x + 5 * p;  // P0, -1/T3, P2, -1/T1, -T2
    double f = c[0] * exp_t(s.T * c[1], s.tab) + c[2] * exp_t(s.T * c[3], s.tab);
    if (t.pm_troe_t2[p]) f += exp_t(c[4] * s.invT, s.tab);
    const double lF = log_t(fmax(f, 1.0e-300), s.ltab) * INV_LN10;
    const double A = lP - 0.67 * lF - 0.4;
    const double B = 0.806 - 1.1762 * lF - 0.14 * lP;
    // log10 F = log10 Fcent / (1 + A^2/B^2) = log10 Fcent B^2 / (B^2 + A^2):
    // one division
    const double B2 = B * B;
    F = exp_t(LN10 * lF * B2 / fma(A, A, B2), s.tab);
  } else {
    const double *c = t.sri_x + 5 * p;  // a, -b, -1/c, d, e
    const double X = 1.0 / (1.0 + lP * lP);
    const double base = c[0] * exp_t(c[1] * s.invT, s.tab) + exp_t(s.T * c[2], s.tab);
    F = exp_t(X * log_t(base, s.ltab), s.tab);
    if (t.pm_sri_de[p]) F *= c[3] * exp_t(c[4] * s.logT, s.tab);
  }
  return low ? F * Pr * inv1p : F * inv1p;
}

// Net rate (fwd - rev) * pres_mod of any reaction: general rate forms,
// pressure modification, non-integer coefficients.
template <class CS, class KC>
__device__ __forceinline__ double rxn_net(const Tab &t, int r, const State &s,
                                          double mix, const CS &C, const KC &kc,
                                          double &fwd, double &rev, double &pm) {
  double xf = 0.0;
  const double kf = rate(t, r, s, xf);
  fwd = kf * product(t.rx_sp, t.rx_nint, t.rx_nu, t.rx_ptr[r], t.rx_ptr[r + 1], C);
  const int j = t.rev_idx[r];
  double net = fwd;
  rev = 0.0;
  if (j >= 0) {
    const double gsum = kc(t, r, j);
    const double kr = (t.rate_kind[r] == RATE_EXP) ? exp_t(xf - gsum, s.tab)
                                                   : kf * exp_t(-gsum, s.tab);
    rev = kr * product(t.px_sp, t.px_nint, t.px_nu, t.px_ptr[r], t.px_ptr[r + 1], C);
    net = fwd - rev;
  }
  const int p = t.pm_idx[r];
  pm = 1.0;
  if (p >= 0) {
    pm = pres_mod(t, p, s, mix, C);
    net *= pm;
  }
  return net;
}

}  // namespace fast
}  // namespace crs
