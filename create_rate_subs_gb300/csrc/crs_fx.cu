// CRS_MODE_FP64: wdot by tiles of 32 states in 64-bit fixed point and FP64.
//
// What bounds it.  The FP64 pipe retires one warp instruction per SM sub-
// partition in ~70 clocks, so 15,000 FP64 instructions per state (53
// species / 325 reactions) held the one-state-per-thread kernel at 33.6 M
// states/s, 95% of that pipe.  Of the arithmetic here FP64 keeps the sums:
// the mass fractions in the reference's order, third bodies, forward minus
// reverse, and one addition per net stoichiometric coefficient, ~2,000 in
// all.  Everything multiplicative -- rate constants, equilibrium constants,
// concentrations, fall-off -- is an exponent in 64-bit fixed point
// (crs_fx.cuh): a product of factors is a sum of integers, a rate constant
// a dot product of a reaction's coefficients with functions of T that are
// formed once per state, and each rate one table exponential.
//
// A reaction's exponents.  On a temperature interval (bounded by 200 K, the
// mechanism's common T_common and 6000 K) with centre and half width of
// log2 T, 1/T and T, the functions L, I, t, t^2, t^3, t^4 are normalised to
// [-1, 1] and every exponent is c0 + cL L + cI I + c1 t + ... + c4 t^4: three
// coefficients forward; the reverse rate's exponent, forward minus ln Kc
// with the Gibbs polynomials of all its species, has seven.  Coefficients
// are rounded to 2^-52, the functions to 2^-61.
//
// A tile: lane = state; the CTA's NW warps share the tile's exponents of
// the concentrations ([N][32], 8 bytes each) and split first the species,
// then the reactions (lists balanced at load by instruction counts), then
// the species sums.  The net rates pass between the last two in shared
// memory or in scratch of one tile per CTA, which stays in L2: without them
// on chip three CTAs share an SM, so that one's sums (FP64 pipe) overlap
// another's rates (integer pipes).  A warp's reaction records stream through
// its own ring of three slots in shared memory, two plain reversible
// reactions at a time, so that their two chains interleave; the next tile's
// mass-fraction sums, two chains of N dependent FP64 additions, run on
// two warps beside the rates.
//
// Measured on GB300 (before: one state per thread, 561/2539 in two passes):
// 2^20 states of 53/325 31.2 -> 6.43 ms, 97 states 716 -> 21.9 us, 20,011
// states of 561/2539 4.87 -> 1.31 ms; FP64 pipe 58%, integer multiply pipe
// 51% busy.
//
// States outside the scheme (T outside (200, 6000] K, a density beyond 2^+-60, a
// mean 1/W out of range, |Y| >= 2, a subnormal Y) and reactions outside it (non-
// integer coefficients, PLOG, Chebyshev, coefficients beyond the bounds)
// are evaluated lane by lane by the general FP64 arithmetic (finish).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "crs_fast.cuh"
#include "crs_fx.cuh"
#include "crs_fx_tab.cuh"
#include "crs_internal.cuh"
#include "crs_tile.cuh"

namespace crs {
namespace fx {

constexpr int64_t ZMIN = -561023779885736503LL;   // log2 1e-300

// The lane's functions of T.
struct Basis {
  Dg L, I, t1, t2, t3, t4;
};
// Rows of a tile's block of per-state values: the six functions, log2 rho,
// y_N, rho, sum Y / W, and two marks: the interval (-1: T outside the scheme)
// and whether the state's sums or fractions are outside it.
constexpr int ROWS = 11;

__device__ __forceinline__ Dg dg(int2 v) { return Dg{v.x, v.y}; }
__device__ __forceinline__ int64_t word(int hi, int lo) {
  return (int64_t)(((uint64_t)(unsigned)hi << 32) | (unsigned)lo);
}
__device__ __forceinline__ int64_t word(int2 v) { return word(v.x, v.y); }

// c0 + sum of coefficient x function; c0 carries the 1 that rounds to even
struct Dot {
  int64_t hh, mid;
  __device__ __forceinline__ explicit Dot(int64_t c0) : hh(c0), mid(1LL << 31) {}
  __device__ __forceinline__ void add(Dg c, Dg f) {
    // (a long sum of products, left to the compiler to fuse)
    hh += (int64_t)c.hi * f.hi;
    mid += (int64_t)c.hi * f.lo;
    mid += (int64_t)c.lo * f.hi;
  }
  __device__ __forceinline__ int64_t exponent() const { return (hh + (mid >> 32)) & ~1LL; }
};

// log2 of a fall-off factor from lth = log2 [M] (c: its record on the lane's
// interval).  slow: outside the scheme (a negative collider or centre, see
// Sum::outside).
__device__ __forceinline__ int64_t falloff(const int2 *__restrict__ c, int flags, int64_t lth,
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
  if (flags & (PMF_TROE | PMF_SRI)) {
    const int64_t zP = z > ZMIN ? z : ZMIN;
    // Fcent (Troe) or the base of the SRI power
    Sum S;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (flags & (PMF_T1 << q)) {
        const int64_t y = word(c[3 + 2 * q]);
        exp2m(y + mul<0>(dg(c[4 + 2 * q]), q == 2 ? I : t), et, M, E);
        S.add(M, E, y & 1);
      }
    }
    slow |= S.outside();
    const int64_t zF = S.log2(lt);
    bool ok;
    f += broadening(zF, zP, flags & PMF_TROE, ok);
    slow |= !ok;
    if (flags & PMF_DE) {
      Dot e(word(c[9]));
      e.add(dg(c[10]), L);
      f += e.exponent();
    }
  }
  // (without its collider a rate in the low-pressure limit is zero)
  if ((flags & PMF_LOW) && lth == ZERO_EXP) f = FALL_MIN_EXP;
  slow |= f < FALL_MIN_EXP;
  return even(f);
}

// Concentrations of one state: on chip, where a state outside the scheme may have
// them in place of its exponents, or from its mass fractions.
struct StateConc {
  const double *conc;  // the state's column, or NULL
  const double *Y;
  int64_t ld;
  double rho, yN;
  const double *inv_mw;
  int N;
  __device__ double operator[](int k) const {
    if (conc) return conc[k * 32];
    return (k == N - 1 ? yN : Y[(int64_t)k * ld]) * (rho * inv_mw[k]);
  }
};

// Stands in a rate's place until the general FP64 arithmetic has formed it, as
// any NaN does (net_of): the loops that form the others then hold no call.
constexpr uint64_t LATER = 0x7ff8000000000000ull;
__device__ __forceinline__ bool is_later(double v) {
  return (bits_of(v) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
}

// The normalised functions of T of one state into column `lane` of the
// block; returns the temperature interval.  irr: T outside the scheme.
__device__ __forceinline__ int basis_of(const FxTab &f, const unsigned char *tab, double T,
                                        int64_t *blk, bool &irr) {
  irr = !(T > f.tb[0] && T <= f.tb[NI]);
  const double Tc = irr ? 1000.0 : T;
  const int iv = Tc > f.tb[1];
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
  const unsigned char *tab;  // fixed-point tables
  const unsigned char *img;  // table image (general FP64 arithmetic)
  double *q;                 // [slots][R + 1][32] scratch when QS is false
  int *busy, slots;          // (tile::claim_slot)
  int list;                  // the work list for NW CL warps
};

// A reaction's record in shared memory: its head and the coefficients of
// the lane's interval.
struct Rec {
  const unsigned char *p, *c;
  __device__ __forceinline__ int4 word4(int o) const {
    return *reinterpret_cast<const int4 *>(p + o);
  }
  __device__ __forceinline__ int4 coef(int u) const {
    return reinterpret_cast<const int4 *>(c)[u];
  }
};

// Copies of a warp's next records into its ring of D slots.
template <int D>
struct Ring {
  const unsigned char *src;
  unsigned base;
  int stride, n, lane;
  // record p (an empty group past the last one)
  __device__ __forceinline__ void fill(int p) const {
    if (p < n) {
      const unsigned char *from = src + (int64_t)p * stride;
      const unsigned to = base + (unsigned)((p % D) * stride);
#pragma unroll 1
      for (int o = lane * 16; o < stride; o += 512)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + o), "l"(from + o)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void start() const {
#pragma unroll
    for (int p = 0; p < D - 1; ++p) fill(p);
  }
  // Record p is on chip for the whole warp; the copy of record p + D - 1
  // starts (its slot's reader, record p - 1, is done).
  __device__ __forceinline__ void next(int p) const {
    __syncwarp();
    fill(p + D - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
    __syncwarp();
  }
};
constexpr int DP = 3, DO = 3;  // slots for pairs of plain records and for other records

__host__ __device__ inline int ring_bytes(const FxTab &f) {
  return f.stride[0] * DP > f.stride[1] * DO ? f.stride[0] * DP : f.stride[1] * DO;
}

// log2 v, bit 0 its sign; zero: ZERO_EXP
__device__ __forceinline__ int64_t log2s(double v, const int64_t *lt) {
  const int64_t l = even(log2d(v, lt)) | (int64_t)(bits_of(v) >> 63);
  return v == 0.0 ? ZERO_EXP : l;
}

// Exponents of the forward and the reverse rate constant.
__device__ __forceinline__ int64_t exponent3(const Rec &r, const Basis &B) {
  const int4 c0 = r.coef(0);
  const int2 c1 = reinterpret_cast<const int2 *>(r.c)[2];
  Dot a(word(c0.x, c0.y));
  a.add(Dg{c0.z, c0.w}, B.L);
  a.add(dg(c1), B.I);
  return a.exponent();
}
__device__ __forceinline__ int64_t exponent7(const Rec &r, const Basis &B) {
  const int2 c0 = reinterpret_cast<const int2 *>(r.c)[3];
  const int4 c1 = r.coef(2), c2 = r.coef(3), c3 = r.coef(4);
  Dot d(word(c0));
  d.add(Dg{c1.x, c1.y}, B.L);
  d.add(Dg{c1.z, c1.w}, B.I);
  d.add(Dg{c2.x, c2.y}, B.t1);
  d.add(Dg{c2.z, c2.w}, B.t2);
  d.add(Dg{c3.x, c3.y}, B.t3);
  d.add(Dg{c3.z, c3.w}, B.t4);
  return d.exponent();
}

// Loads of one tile's mass fractions (rows of this warp) straight into
// shared memory; row N - 1 is y_N.
template <int NW>
__device__ __forceinline__ void load_y(const double *Y, int64_t ld, int N, int warp,
                                       unsigned smem_rows) {
#pragma unroll 4
  for (int k = warp; k < N - 1; k += NW)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_rows + k * 256),
                 "l"(Y + (int64_t)k * ld)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// y_N = 1 - sum y in the reference's order (rate_subs.py:1312-1320) on warp
// 0, sum y / W and the density on warp 1: two dependent FP64 chains side by
// side.  Rows 6.. of the block: log2 rho, y_N, rho, sum y / W.
__device__ __forceinline__ void state_sums(const double *Y, int64_t ld, int N, int warp,
                                           const double *inv_mw, double T, double P,
                                           const int64_t *lt, double *row, int *irr) {
  if (warp == 0) {
    double ys = N > 1 ? Y[0] : 0.0;
    int k = 1;
    for (; k + 8 <= N - 1; k += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = Y[(int64_t)(k + u) * ld];
#pragma unroll
      for (int u = 0; u < 8; ++u) ys += v[u];
    }
    for (; k < N - 1; ++k) ys += Y[(int64_t)k * ld];
    row[7 * 32] = 1.0 - ys;
    asm volatile("bar.sync 1, 64;" ::: "memory");
  } else if (warp == 1) {
    double mwi = 0.0;
    int k = 0;
    for (; k + 8 <= N - 1; k += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = Y[(int64_t)(k + u) * ld];
#pragma unroll
      for (int u = 0; u < 8; ++u) mwi = fma(v[u], inv_mw[k + u], mwi);
    }
    for (; k < N - 1; ++k) mwi = fma(Y[(int64_t)k * ld], inv_mw[k], mwi);
    asm volatile("bar.sync 1, 64;" ::: "memory");
    mwi = fma(row[7 * 32], inv_mw[N - 1], mwi);
    const double rho = P / mwi * ((1.0 / T) * fast::INV_RU);
    // a positive density of moderate size (RHO_MAX), a mean 1/W below 2
    const int e = (int)(bits_of(rho) >> 52), m = (int)(bits_of(mwi) >> 52);
    *irr = e < 1023 - RHO_MAX || e >= 1023 + RHO_MAX || m < 1023 - 40 || m > 1023;
    reinterpret_cast<int64_t *>(row)[6 * 32] = even(log2d(rho, lt));
    row[8 * 32] = rho;
    row[9 * 32] = mwi;
  }
}

// Functions of T, sums and marks of one tile's states into the block at o
// (warps 0-2; i: the lane's state).  Called, not inlined: once per tile, and
// its registers are not the rate loops'.
__device__ __noinline__ void prepare(const FxTab &f, const Args &g, const double *inv_mw,
                                     const Batch &b, int64_t i, int warp, int lane,
                                     const int64_t *lt, unsigned char *o) {
  int *marks = reinterpret_cast<int *>(o + 10 * 256 - lane * 8) + lane;
  if (warp == 2) {
    bool irr;
    const int iv = basis_of(f, g.tab, b.T[i], reinterpret_cast<int64_t *>(o), irr);
    marks[0] = irr ? -1 : iv;
  } else if (warp < 2) {
    state_sums(b.Y + i, b.ld, f.N, warp, inv_mw, b.T[i], b.P[i], lt,
               reinterpret_cast<double *>(o), marks + 32);
  }
}

// Rates left to the general FP64 arithmetic: one state's (i), of the warp's
// records (all: every one, else those marked; conc: its concentrations on chip).
// SPREAD: of records first, first + step, ...; else of all, or none if step is 0.
template <bool SPREAD>
__device__ __noinline__ void finish(const Args &g, const ImgLayout &lay, const Batch &b,
                                    int stride, Ring<DP> plain, Ring<DO> other, int64_t i,
                                    bool all, const double *conc, double rho, double yN,
                                    unsigned char *q, int first, int step) {
  const Tab t = make_tab(g.img, lay);
  fast::State s;
  s.T = b.T[i];
  s.P = b.P[i];
  s.invT = 1.0 / s.T;
  s.logT = fast::log_t(s.T, t.logtab);
  s.tab = t.exptab;
  s.ltab = t.logtab;
  KcPolyG kc;
  kc.T = s.T;
  kc.logT = s.logT;
  kc.invT = s.invT;
  const StateConc C{conc, b.Y + i, b.ld, rho, yN, t.inv_mw, t.N};
  const int n = SPREAD || step ? 2 * plain.n + other.n : 0;
#pragma unroll 1
  for (int p = SPREAD ? first : 0; p < n; p += SPREAD ? step : 1) {
    const int o = p - 2 * plain.n;
    const int4 h = __ldg(reinterpret_cast<const int4 *>(
        o < 0 ? plain.src + (int64_t)p * stride : other.src + (int64_t)o * other.stride));
    double *v = reinterpret_cast<double *>(q + h.x);
    double fwd, rev, pm;
    if (h.w >= 0 && (all || is_later(*v)))
      *v = fast::rxn_net(t, h.w, s, s.P * s.invT * fast::INV_RU, C, kc, fwd, rev, pm);
  }
}

// FP64 concentrations in place of the exponents, for a lane whose state i is
// outside the scheme (o: its column of the block).
__device__ __noinline__ void concentrations(const Batch &b, const double *inv_mw, int64_t i, int N,
                                            int warp, int nw, const unsigned char *o,
                                            unsigned char *yl) {
  const double yN = *reinterpret_cast<const double *>(o + 7 * 256);
  const double rho = *reinterpret_cast<const double *>(o + 8 * 256);
#pragma unroll 1
  for (int k = warp; k < N; k += nw)
    *reinterpret_cast<double *>(yl + k * 256) =
        (k == N - 1 ? yN : b.Y[(int64_t)k * b.ld + i]) * (rho * inv_mw[k]);
}

// A warp's lists, entry 0..6: its first plain record and the next warp's, its
// first other record and the next warp's, its first species and the next warp's,
// its first group of terms.  ON_CHIP: in shared memory, the registers being short.
template <bool ON_CHIP>
struct Lists {
  int *chip;
  int reg[7];
  __device__ __forceinline__ Lists(const FxTab &f, const unsigned char *tab, int list, int gw,
                                   int *chip_, int lane)
      : chip(chip_) {
    const int at[7] = {f.list_ptr[list][0], f.list_ptr[list][0], f.list_ptr[list][1],
                       f.list_ptr[list][1], f.seg_ptr[list],     f.seg_ptr[list],
                       f.term_ptr[list]};
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      if (!ON_CHIP)
        reg[k] = reinterpret_cast<const int *>(tab + at[k])[gw + (k & 1)];
      else if (lane == k)
        chip[k] = reinterpret_cast<const int *>(tab + at[k])[gw + (k & 1)];
    }
    __syncwarp();
  }
  __device__ __forceinline__ int operator[](int k) const { return ON_CHIP ? chip[k] : reg[k]; }
};

// Barrier of the CTAs that share a tile.
template <int CL>
__device__ __forceinline__ void tile_barrier() {
  if (CL == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// NW warps per CTA, CL CTAs (a cluster) per tile: each forms the tile's
// exponents for itself, evaluates its share of the reactions and, the rates
// exchanged through the first CTA's shared memory (QS) or scratch, of the
// species.
template <int NW, int PER_SM, int CL, bool QS, bool TS>
__global__ void __launch_bounds__(NW * 32, PER_SM)
    k_wdot_tile(const __grid_constant__ ImgLayout lay, const __grid_constant__ FxTab f,
                const __grid_constant__ Args g, const __grid_constant__ Batch b) {
  const int LIST = g.list;
  extern __shared__ __align__(128) unsigned char smem[];
  const int N = f.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned char *tab = g.tab;
  // shared memory: [N + 1][32] y, then the exponents of C (row N: zeros);
  // two blocks of per-state values; the small tables; each warp's ring of
  // records; the warps' lists; the net rates
  unsigned char *yl = smem + lane * 8;
  unsigned char *next = smem + (N + 1) * 256;
  unsigned char *blk0 = next + lane * 8;
  next += 2 * ROWS * 256;
  const int64_t *et = reinterpret_cast<const int64_t *>(tab + f.small);
  if (TS) {
    int64_t *st = reinterpret_cast<int64_t *>(next);
    for (int k = threadIdx.x; k < TAB_BYTES / 8; k += NW * 32) st[k] = et[k];
    et = st;
    next += TAB_BYTES;
    __syncthreads();
  }
  const int64_t *lt = et + EXP_WORDS;
  const int rb = ring_bytes(f);
  unsigned char *ring = next + warp * rb;
  next += NW * rb;
  // How rates are left to the general arithmetic.  SPREAD: the lanes may share
  // them (see there), with the lists on chip to have the registers.  OUTS: whole
  // tiles outside the scheme go there at once, and such states' concentrations are
  // on chip.  Both cost the loops registers.  With 24 warps none is missed (8,192
  // states of 561/2539, all outside: 2.84 -> 2.23 ms, one in 97: 2.85 -> 0.80);
  // with 8 OUTS took 1% and SPREAD 4% (2^18 states of 53/325, all outside: 10.1 ->
  // 7.86 ms with OUTS, one in 97: 4.9 -> 4.3); with 16, for few tiles, where
  // latency counts, both would take 4% (4,000 states 45.3 -> 47.2 us).
  constexpr bool SPREAD = NW == 24, OUTS = NW != 16;
  int *chip = reinterpret_cast<int *>(next) + warp * 8;
  if (SPREAD) next += NW * 32;
  __shared__ int s_slot;
  if (!QS && blockIdx.x % CL == 0 && threadIdx.x == 96)  // for the CTAs of the tile
    s_slot = tile::claim_slot(g.busy, g.slots, blockIdx.x / CL, b.status);
  unsigned char *q = (QS && CL > 1 ? static_cast<unsigned char *>(__cluster_map_shared_rank(next, 0))
                                   : next) + lane * 8;  // (scratch: once there is a slot)
  auto Yl = [&](int off) -> int64_t & { return *reinterpret_cast<int64_t *>(yl + off); };
  auto Q = [&](int off) -> double & { return *reinterpret_cast<double *>(q + off); };
  if (warp == 0) {
    Yl(N * 256) = 0;
    if (QS) reinterpret_cast<double *>(next)[f.R * 32 + lane] = 0.0;  // before all CTAs run
  }
  const int gw = CL == 1 ? warp : (int)(blockIdx.x % CL) * NW + warp;  // the tile's warp
  const Lists<SPREAD> lists(f, tab, LIST, gw, chip, lane);
  auto plain_of = [&] {
    return Ring<DP>{tab + f.rec[LIST][0] + (int64_t)lists[0] * f.stride[0], smem_u32(ring),
                    f.stride[0], lists[1] - lists[0], lane};
  };
  auto other_of = [&] {
    return Ring<DO>{tab + f.rec[LIST][1] + (int64_t)lists[2] * f.stride[1], smem_u32(ring),
                    f.stride[1], lists[3] - lists[2], lane};
  };
  auto terms_of = [&] {
    return reinterpret_cast<const int4 *>(tab + f.term[LIST]) + lists[6];
  };
  const Ring<DP> plain_kept = plain_of();
  const Ring<DO> other_kept = other_of();
  const int4 *terms_kept = terms_of();
  auto plain_list = [&] { return SPREAD ? plain_of() : plain_kept; };
  auto other_list = [&] { return SPREAD ? other_of() : other_kept; };
  const unsigned yrows = smem_u32(smem) + lane * 8;
  const double *inv_mw = reinterpret_cast<const double *>(g.img + lay.inv_mw);
  int bad = 0, bk = 0;
  int64_t tile = blockIdx.x / CL;
  const int64_t step = gridDim.x / CL;
  const int64_t ntiles = (b.n + 31) / 32;
  if (tile < ntiles) {
    const int64_t i = tile * 32 + lane < b.n ? tile * 32 + lane : tile * 32;
    load_y<NW>(b.Y + i, b.ld, N, warp, yrows);
    if (warp < 3) prepare(f, g, inv_mw, b, i, warp, lane, lt, blk0);
  }
  if (!QS) {  // (the claim ran beside the first tile's sums)
    tile_barrier<CL>();
    const int slot =
        CL > 1 ? *static_cast<const int *>(__cluster_map_shared_rank(&s_slot, 0)) : s_slot;
    q = reinterpret_cast<unsigned char *>(g.q) + (int64_t)slot * (f.R + 1) * 256 + lane * 8;
    if (warp == 0) Q(f.R * 256) = 0.0;
  }
  for (; tile < ntiles; tile += step, bk ^= 1) {
    const int64_t i = tile * 32 + lane;
    const bool valid = i < b.n;
    const int64_t ic = valid ? i : tile * 32;  // idle lanes repeat a valid state
    asm volatile("cp.async.wait_all;" ::: "memory");
    tile_barrier<CL>();
    unsigned char *o = blk0 + bk * ROWS * 256;
    auto rowd = [&](int r) { return *reinterpret_cast<const double *>(o + r * 256); };
    int *marks = reinterpret_cast<int *>(o + 10 * 256 - lane * 8) + lane;
    const int64_t lrho = *reinterpret_cast<const int64_t *>(o + 6 * 256);
    // a third-body concentration over rho: 1/mw + sum (eff - 1) Y / W
    auto third_body = [&](int p) {
      const int *ep = reinterpret_cast<const int *>(tab + f.eff_ptr) + p;
      double s = rowd(9);
      auto term = [&](int e, double &c) {
        const int4 w = __ldg(reinterpret_cast<const int4 *>(tab + f.eff) + e);
        c = __hiloint2double(w.y, w.x);
        return w.z == (N - 1) * 256 ? rowd(7)
               : QS && CL == 1      ? __longlong_as_double(Yl(w.z))
                                    : b.Y[(int64_t)(w.z >> 8) * b.ld + ic];
      };
      // the loads of a group of terms ahead of its chain of additions, where
      // one CTA's latency shows (97 states of 53/325: 22.5 -> 21.6 us, 65,536
      // of 561/2539: 4.45 -> 4.41 ms); with more CTAs per SM the registers
      // count (2^20 states of 53/325: 6.41 -> 6.50 ms)
      int e = __ldg(ep);
      const int e1 = __ldg(ep + 1);
      if constexpr (PER_SM == 1) {
#pragma unroll 1
        for (; e + 4 <= e1; e += 4) {
          double c[4], y[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) y[u] = term(e + u, c[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u) s = fma(c[u], y[u], s);
        }
      }
#pragma unroll 1
      for (; e < e1; ++e) {
        double c;
        const double y = term(e, c);
        s = fma(c, y, s);
      }
      return s;
    };
    // (rates on chip) into the slots of their reactions' rates
    if (QS && CL == 1 && f.NPM > 0) {
#pragma unroll 1
      for (int p = warp; p < f.NPM; p += NW) {
        const int slot = __ldg(reinterpret_cast<const int2 *>(tab + f.pm) + p).x;
        if (slot >= 0) Q(slot) = third_body(p);
      }
      __syncthreads();
    }
    // exponents of the concentrations in place of the mass fractions
    bool odd = false;
#pragma unroll 1
    for (int k = warp; k < N; k += NW) {
      const double y = k == N - 1 ? rowd(7) : __longlong_as_double(Yl(k * 256));
      const uint64_t u = bits_of(y);
      const int e = (int)(u >> 52) & 0x7ff;
      int64_t l = even(log2d(y, lt) + reinterpret_cast<const int64_t *>(tab + f.lw)[k] + lrho) |
                  (int64_t)(u >> 63);
      const bool zero = (u << 1) == 0;
      if (zero) l = ZERO_EXP;
      odd |= !zero && (e == 0 || e > 1023);  // subnormal, |y| >= 2, NaN
      Yl(k * 256) = l;
    }
    if (odd) marks[32] = 1;
    plain_list().start();
    __syncthreads();
    // net rates
    {
      if (warp < 3 && tile + step < ntiles) {
        const int64_t j = (tile + step) * 32;
        prepare(f, g, inv_mw, b, j + lane < b.n ? j + lane : j, warp, lane, lt,
                blk0 + (bk ^ 1) * ROWS * 256);
      }
      const int iv = marks[0] < 0 ? 0 : marks[0];
      // states outside the scheme: every rate in FP64, from concentrations in
      // place of their exponents; later: single rates
      const bool out = marks[0] < 0 || marks[32];
      bool later = false;
      if (OUTS && __any_sync(0xffffffffu, out)) {  // (the tile's marks: for all warps)
        if (out) concentrations(b, inv_mw, ic, N, warp, NW, o, yl);
        __syncthreads();
      }
      Basis B;
      B.L = dg(*reinterpret_cast<const int2 *>(o));
      B.I = dg(*reinterpret_cast<const int2 *>(o + 256));
      B.t1 = dg(*reinterpret_cast<const int2 *>(o + 512));
      B.t2 = dg(*reinterpret_cast<const int2 *>(o + 768));
      B.t3 = dg(*reinterpret_cast<const int2 *>(o + 1024));
      B.t4 = dg(*reinterpret_cast<const int2 *>(o + 1280));
      // the record at `at` whose coefficients begin `co` bytes on
      auto record = [&](const unsigned char *at, int co) {
        int idx = iv;
        if (f.nthr) {
          const double T = b.T[ic];
          const double *thr = reinterpret_cast<const double *>(at + co + COEF * (f.nthr + 1));
          idx = 0;
  #pragma unroll 1
          for (int e = 0; e < f.nthr; ++e) idx += T > thr[e];
        }
        return Rec{at, at + co + COEF * idx};
      };
      const int one = f.stride[0] / 2;
      const bool skip = OUTS && __all_sync(0xffffffffu, out);  // a whole tile outside
      // two reactions at a time: independent chains side by side
      const Ring<DP> plain = plain_list();
      unsigned char *at = ring;
#pragma unroll 1
      for (int p = skip ? plain.n : 0; p < plain.n; ++p) {
        plain.next(p);
        int64_t yf[2], yr[2];
        int slot[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const Rec r = record(at + u * one, HEAD);
          const int2 h = *reinterpret_cast<const int2 *>(r.p);  // slot, flags
          const int4 x = r.word4(16);
          slot[u] = h.x;
          yf[u] = (exponent3(r, B) | (h.y & RF_NEG)) + Yl(x.x) + Yl(x.y);
          yr[u] = (exponent7(r, B) | (h.y & RF_NEG)) + Yl(x.z) + Yl(x.w);
          if (h.y & RF_MORE) {
            const int4 m = r.word4(32);
            yf[u] += Yl(m.x) + Yl(m.y);
            yr[u] += Yl(m.z) + Yl(m.w);
          }
        }
        bool far[2];
        const double v0 = net_of<true>(yf[0], yr[0], et, far[0]);
        const double v1 = net_of<true>(yf[1], yr[1], et, far[1]);
        Q(slot[0]) = v0;
        Q(slot[1]) = v1;
        later |= far[0] | far[1];
        at = at == ring + 2 * f.stride[0] ? ring : at + f.stride[0];
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      const Ring<DO> other = other_list();
      other.start();
#pragma unroll 1
      for (int p = skip ? other.n : 0; p < other.n; ++p) {
        other.next(p);
        const Rec r = record(ring + (p % DO) * f.stride[1], HEAD + PMH + PMC * NI);
        const int4 h = r.word4(0), x = r.word4(16), ph = r.word4(HEAD);
        bool slow = h.y & RF_GEN;
        int64_t l = h.y & RF_NEG;  // what both directions share
        double thd = 1.0;
        if (h.z >= 0) {
          if (h.y & RF_FALL) {
            const int64_t lth = ph.y >= 0
                                    ? Yl(ph.y)
                                    : log2s(QS && CL == 1 ? Q(h.x) : third_body(h.z), lt) + lrho;
            l += falloff(reinterpret_cast<const int2 *>(r.p + HEAD + PMH + PMC * iv), ph.x, lth,
                         B.L, B.I, B.t1, et, lt, slow);
          } else {
            thd = rowd(8) * (QS && CL == 1 ? Q(h.x) : third_body(h.z));
          }
        }
        int64_t yf = exponent3(r, B) + l + Yl(x.x) + Yl(x.y);
        const int4 m = r.word4(32);
        yf += Yl(m.x) + Yl(m.y);
        double v;
        bool far;
        if (h.y & RF_REV) {
          const int64_t yr = exponent7(r, B) + l + Yl(x.z) + Yl(x.w) + Yl(m.z) + Yl(m.w);
          v = net_of<true>(yf, yr, et, far);
        } else {
          v = net_of<false>(yf, 0, et, far);
        }
        slow |= far;
        Q(h.x) = slow ? of_bits(LATER) : v * thd;
        later |= slow;
      }
      // What is left: lane = state or, for few states, lane = reaction, state by
      // state, in as many turns as there are records for 32 lanes, each with the
      // code of several kinds of reactions (2.5 times one's).
      if (SPREAD) {
        if (unsigned need = __ballot_sync(0xffffffffu, later || out)) {
          const Ring<DP> plain = plain_list();
          const Ring<DO> other = other_list();
          const int n = 2 * plain.n + other.n;
          const bool spread = 5 * __popc(need) * ((n + 31) / 32) < 2 * n;
          if (!spread) need = 1u;
          __syncwarp();  // the marks of the other lanes
          do {
            const int src = spread ? __ffs(need) - 1 : lane, off = (src - lane) * 8;
            const bool all = __shfl_sync(0xffffffffu, (int)out, src);
            const int64_t is = __shfl_sync(0xffffffffu, ic, src);
            const double rho = __shfl_sync(0xffffffffu, rowd(8), src);
            const double yN = __shfl_sync(0xffffffffu, rowd(7), src);
            if (spread || later || out)
              finish<true>(g, lay, b, one, plain, other, is, all,
                           all ? reinterpret_cast<double *>(yl + off) : nullptr, rho, yN, q + off,
                           spread ? lane : 0, spread ? 32 : 1);
            __syncwarp();
            need &= need - 1;
          } while (need);
        }
      } else if (__any_sync(0xffffffffu, later || out)) {
        finish<false>(g, lay, b, one, plain_kept, other_kept, ic, out,
                      OUTS && out ? reinterpret_cast<double *>(yl) : nullptr, rowd(8), rowd(7), q,
                      0, later || out);
      }
    }
    // the first terms are on their way before the barrier
    const int s0 = lists[4], s1 = lists[5];
    const int4 *terms = SPREAD ? terms_of() : terms_kept;
    const int4 t0 = __ldg(terms), t1 = __ldg(terms + 1);
    const int4 sg0 = __ldg(reinterpret_cast<const int4 *>(tab + f.seg[LIST]) + s0);
    tile_barrier<CL>();
    // the next tile's mass fractions replace exponents that every warp is
    // done with, while the species sums run
    if (tile + step < ntiles) {
      const int64_t j = (tile + step) * 32;
      load_y<NW>(b.Y + (j + lane < b.n ? j + lane : j), b.ld, N, warp, yrows);
    }
    {
      // the groups of the warp's species are one stream: the rates of the
      // next group are on their way while a group is added
      auto rates = [&](int4 t, double (&v)[4]) {
        const int x[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double d = Q(x[u] & 0x7fffffff);
          v[u] = __hiloint2double(__double2hiint(d) ^ (x[u] & 0x80000000), __double2loint(d));
        }
      };
      const int4 *tm = terms;
      double v[4];
      rates(t0, v);
      int4 t = t1, sgn = sg0;
#pragma unroll 1
      for (int a = s0; a < s1; ++a) {
        const int4 sg = sgn;
        sgn = __ldg(reinterpret_cast<const int4 *>(tab + f.seg[LIST]) + a + 1);
        double w = 0.0, w2 = 0.0;
#pragma unroll 1
        for (int e = 0; e < sg.y; ++e) {
          double u[4];
          rates(t, u);
          t = __ldg(tm + 2);
          ++tm;
          w += v[0];
          w2 += v[1];
          w += v[2];
          w2 += v[3];
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c] = u[c];
        }
#pragma unroll 1
        for (int e = sg.z; e < sg.z + sg.w; ++e)
          w = fma(__ldg(reinterpret_cast<const double *>(tab + f.wnu) + e),
                  Q(__ldg(reinterpret_cast<const int *>(tab + f.wterm) + e)), w);
        w += w2;
        if (valid) {
          bad += ((__double2hiint(w) >> 20) & 0x7ff) == 0x7ff;  // inf or NaN, integer test
          b.wdot[(int64_t)sg.x * b.ld + i] = w;
        }
      }
    }
    // rates are replaced only after the barrier at the loop's head
  }
  if (!QS || CL > 1) tile_barrier<CL>();  // the tile's rates are read until here
  if (!QS && blockIdx.x % CL == 0 && threadIdx.x == 0)
    tile::release_slot(g.busy, g.slots, s_slot);
  if (bad && b.status) atomicAdd(&b.status[1], bad);
}

// Shared memory of a CTA of nw warps.
size_t smem_of(const FxTab &f, int nw, bool qs, bool ts) {
  return (size_t)(f.N + 1 + 2 * ROWS) * 256 + (ts ? TAB_BYTES : 0) +
         (size_t)nw * (ring_bytes(f) + 32) + (qs ? (size_t)(f.R + 1) * 256 : 0);
}

// How a launch over `tiles` tiles runs: warps per CTA, CTAs per SM and per
// tile, rates and small tables on chip.
struct Plan {
  int nw = 24, per_sm = 1, cl = 1;
  bool qs = false, ts = false, ok = false;
};

Plan plan_of(const FxTab &f, int64_t tiles, int sm_count, int smem_optin) {
  if (!f.usable) return Plan{};
  auto fits = [&](int nw, int per_sm, bool qs) {
    return (smem_of(f, nw, qs, true) + 1024) * per_sm <= (size_t)smem_optin + 1024;
  };
  // few tiles: a cluster of CTAs shares each, as long as its warps get two
  // reactions or more (97 states of 53/325: 47 us with one CTA per tile, 21.6
  // with eight)
  for (int cl = 8; cl > 1; cl /= 2)
    if (tiles * cl <= sm_count && f.R >= 32 * cl) {
      if (fits(16, 1, true)) return Plan{16, 1, cl, true, true, true};
      if (fits(16, 1, false)) return Plan{16, 1, cl, false, true, true};
    }
  // one tile per SM: its rates on chip, more warps (4,000 states of 53/325:
  // 57 us with three CTAs of eight warps, 45 so)
  if (tiles <= sm_count && fits(16, 1, true)) return Plan{16, 1, 1, true, true, true};
  // small mechanisms: a tile's work does not fill more warps (131,072 states
  // of 10/27: 115 us with three CTAs of eight, 101 so)
  if (f.R < 100 && fits(4, 6, true)) return Plan{4, 6, 1, true, true, true};
  // rates in L2, so that three CTAs share an SM and their phases overlap (2^20
  // states of 53/325: 6.41 ms; rates on chip, one CTA of 16 warps: 8.5; six
  // CTAs of four: 6.89)
  if (fits(8, 3, false)) return Plan{8, 3, 1, false, true, true};
  if (fits(24, 1, false)) return Plan{24, 1, 1, false, true, true};
  Plan p{24, 1, 1, false, false, false};
  p.ok = smem_of(f, 24, false, false) <= (size_t)smem_optin;
  return p;
}

using Kernel = void (*)(const ImgLayout, const FxTab, const Args, const Batch);
Kernel kernel_of(const Plan &p) {
  switch (p.cl) {
    case 8: return p.qs ? k_wdot_tile<16, 1, 8, true, true> : k_wdot_tile<16, 1, 8, false, true>;
    case 4: return p.qs ? k_wdot_tile<16, 1, 4, true, true> : k_wdot_tile<16, 1, 4, false, true>;
    case 2: return p.qs ? k_wdot_tile<16, 1, 2, true, true> : k_wdot_tile<16, 1, 2, false, true>;
  }
  if (p.nw == 4) return k_wdot_tile<4, 6, 1, true, true>;
  if (p.nw == 16) return k_wdot_tile<16, 1, 1, true, true>;
  if (p.nw == 8) return k_wdot_tile<8, 3, 1, false, true>;
  return p.ts ? k_wdot_tile<24, 1, 1, false, true> : k_wdot_tile<24, 1, 1, false, false>;
}

}  // namespace fx

// Raises the kernels' shared-memory limit to the device's, once per load of a
// mechanism (a microsecond or two per launch otherwise).
cudaError_t fx_init(int smem_optin) {
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < 7 && e == cudaSuccess; ++q) {
    fx::Plan p;
    p.cl = q < 3 ? 2 << q : 1;
    p.nw = q == 3 ? 4 : q == 4 ? 16 : q == 5 ? 8 : 24;
    p.ts = p.qs = true;
    e = set_smem_limit(fx::kernel_of(p), (size_t)smem_optin);
    p.ts = p.qs = false;
    if (e == cudaSuccess) e = set_smem_limit(fx::kernel_of(p), (size_t)smem_optin);
  }
  return e;
}

// A launch over n states is one or two kernels: whole waves of tiles, and
// what is left over, whose few tiles are shared by clusters (626 tiles of a
// large mechanism on 152 SMs: the fifth wave held 18).  Tiles of the first:
static int64_t first_tiles(const fx::FxTab &f, int64_t tiles, int sm_count, int smem_optin) {
  const fx::Plan p = fx::plan_of(f, tiles, sm_count, smem_optin);
  const int64_t wave = (int64_t)sm_count * p.per_sm;
  const int64_t rest = tiles % wave;
  // worth a launch when two or more CTAs may share each tile
  return p.cl > 1 || tiles < wave || rest == 0 || 2 * rest > sm_count || f.R < 64
             ? tiles
             : tiles - rest;
}

// Whether a launch over n states needs scratch (0: the net rates fit on chip);
// < 0: the mechanism does not fit this kernel.
int fx_scratch(const fx::FxTab &f, int64_t n, int sm_count, int smem_optin) {
  const int64_t tiles = (n + 31) / 32, first = first_tiles(f, tiles, sm_count, smem_optin);
  int need = 0;
  for (int64_t part : {first, tiles - first}) {
    if (part == 0) continue;
    const fx::Plan p = fx::plan_of(f, part, sm_count, smem_optin);
    if (!p.ok) return -1;
    need |= !p.qs;
  }
  return need;
}

// The resources of the launches that need scratch.
cudaError_t fx_slots(const fx::FxTab &f, int sm_count, int smem_optin, SlotUse &u) {
  cudaError_t e = cudaSuccess;
  // every plan: few tiles, one per SM, more
  for (int64_t tiles : {1, sm_count / 8 + 1, sm_count / 4 + 1, sm_count / 2 + 1, sm_count + 1}) {
    const fx::Plan p = fx::plan_of(f, tiles, sm_count, smem_optin);
    if (p.ok && !p.qs && e == cudaSuccess)
      e = u.add(fx::kernel_of(p), p.nw * 32, fx::smem_of(f, p.nw, p.qs, p.ts));
  }
  return e;
}

static cudaError_t launch_tiles(const unsigned char *img, const ImgLayout &L,
                                const fx::FxTab &f, const unsigned char *tab, const Batch &b,
                                int sm_count, int smem_optin, const TileScratch &scratch,
                                cudaStream_t s) {
  const int64_t tiles = (b.n + 31) / 32;
  const fx::Plan p = fx::plan_of(f, tiles, sm_count, smem_optin);
  if (!p.ok || (!p.qs && !scratch.q)) return cudaErrorInvalidValue;
  int list = 0;
  while (list < fx::NLIST - 1 && fx::list_warps[list] != p.nw * p.cl) ++list;
  const fx::Kernel k = fx::kernel_of(p);
  const size_t bytes = fx::smem_of(f, p.nw, p.qs, p.ts);
  const int64_t grid = std::min<int64_t>(tiles, (int64_t)sm_count * p.per_sm) * p.cl;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)p.nw * 32);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = p.cl > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, L, f, fx::Args{tab, img, scratch.q, scratch.busy, scratch.slots, list}, b);
}

cudaError_t launch_wdot_fx(const unsigned char *img, const ImgLayout &L, const fx::FxTab &f,
                           const unsigned char *tab, const Batch &b, int sm_count,
                           int smem_optin, const TileScratch &scratch, cudaStream_t s) {
  const int64_t tiles = (b.n + 31) / 32, first = first_tiles(f, tiles, sm_count, smem_optin);
  Batch part = b;
  part.n = std::min<int64_t>(b.n, first * 32);
  cudaError_t e = launch_tiles(img, L, f, tab, part, sm_count, smem_optin, scratch, s);
  if (e != cudaSuccess || first == tiles) return e;
  const int64_t o = part.n;
  part.n = b.n - o;
  part.T += o;
  part.P += o;
  part.Y += o;
  part.wdot += o;
  return launch_tiles(img, L, f, tab, part, sm_count, smem_optin, scratch, s);
}

}  // namespace crs
