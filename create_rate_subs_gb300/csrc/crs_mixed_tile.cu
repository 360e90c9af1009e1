// CRS_MODE_MIXED by tiles of 32 states: the arithmetic of crs_mixed.cuh in the
// layout of crs_fx.cu.
//
// What bounds it.  The one-state-per-thread kernel holds 11 warps per SM
// (12 bytes of shared memory per species and thread, 168 registers) and
// waits: 42% of its issue slots, 35% of the FP64 pipe.  Here lane = state and
// the warps of a CTA share the tile's concentrations and split its
// reactions, then its species sums, so that 24 warps of 80 registers fit
// whatever the mechanism's size; few tiles are shared by clusters.  Records
// stream through each warp's ring in shared memory, two reactions of one
// shape group at a time.  Three-body and fall-off reactions have records
// too: read through the general tables, with their calls, the 60 of them
// among 53/325 took more than the other 265.
//
// The FP32 operations of a rate from its exponent on are those of the one-
// state-per-thread kernel (a factor of one in place of an absent one is
// exact), so the FP32 roundings are the same; FP64 keeps forward minus
// reverse, concentrations and sums.  What does not change them is done once:
// concentrations are kept as mantissa and exponent, the reverse exponent has
// its own coefficients, and the clamps of an exponential and of a double's
// range are one test of its exponent, behind which the general code stands.
// That took the warp instructions per state from 4,602 to 3,857 and the time
// from 23.7 to 20.9 ms; the FP64 pipe is 65% busy, the schedulers 61%.
//
// Measured on GB300 (before: one state per thread, large mechanisms in two
// passes): 2^22 states of 53/325 35.6 -> 20.9 ms, 65,536 of 561/2539 5.32 ->
// 3.17 ms.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "crs_exp.cuh"
#include "crs_fx_tab.cuh"
#include "crs_internal.cuh"
#include "crs_mixed.cuh"
#include "crs_tile.cuh"

namespace crs {
namespace mixt {

using namespace mixed;
using namespace fx;

struct Args {
  const unsigned char *tab;  // fixed-point tables (lists, records)
  const unsigned char *img;  // table image
  double *q;                 // [slots][R + 1][32] scratch when QS is false
  int *busy, slots;          // (tile::claim_slot)
  int list;                  // the work list for NW CL warps
  // contraction (PACK): bf16 rows [i][2 Kh] and the states' scale exponents
  __nv_bfloat16 *A;
  int Kh;
  int *escale;
};

constexpr int WINDOW = 100;  // binary orders around the scale carried by bf16 hi + lo

__device__ __forceinline__ bool in_window(double v, int c) {
  const int hi = __double2hiint(v), lo = __double2loint(v);
  const int e = (hi >> 20) & 0x7ff;
  const bool zero = ((hi & 0x7fffffff) | lo) == 0;
  return zero || (e != 0 && e != 0x7ff && abs(e - 1023 - c) <= WINDOW);
}

// Sum and count of the binary exponents of the rates that a lane has formed.
struct Scale {
  int sum = 0, count = 0;
  __device__ __forceinline__ void add(double v) {
    const int hi = __double2hiint(v), e = (hi >> 20) & 0x7ff;
    const bool c = e != 0x7ff && ((hi & 0x7fffffff) | __double2loint(v)) != 0;
    sum += c ? e - 1023 : 0;
    count += c;
  }
};

// 32 bytes to a 32-byte aligned address: a whole sector per lane
__device__ __forceinline__ void store32(void *p, const unsigned (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]),
               "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

constexpr int D = 3;  // slots of a warp's ring of pairs of records

// (The ring, the barrier and the sums are crs_fx.cu's in other words: there,
// as functions shared by both kernels, they cost 6.41 -> 6.50 ms for 2^20
// states of 53/325, the registers falling otherwise.)

// Copies of a warp's next records into its ring of D slots.
template <int D>
struct Ring {
  const unsigned char *src;
  unsigned base;
  int stride, n, lane;
  // record p into slot s (an empty group past the last one)
  __device__ __forceinline__ void fill(int p, int s) const {
    if (p < n) {
      const unsigned char *from = src + (unsigned)(p * stride + lane * 16);
      const unsigned to = base + (unsigned)(s * stride + lane * 16);
      if (lane * 16 < stride)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
      if (stride > 512) {
#pragma unroll 1
        for (int o = 512; o < stride - lane * 16; o += 512)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + o), "l"(from + o)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void start() const {
#pragma unroll
    for (int p = 0; p < D - 1; ++p) fill(p, p);
  }
  // Record p, in slot s, is on chip for the whole warp; the copy of record
  // p + D - 1 starts (its slot's reader, record p - 1, is done).  Returns the
  // next record's slot.
  __device__ __forceinline__ int next(int p, int s) const {
    __syncwarp();
    fill(p + D - 1, s == 0 ? D - 1 : s - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
    __syncwarp();
    return s == D - 1 ? 0 : s + 1;
  }
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

// The species sums of one warp (gw of list `list`) of a tile: each species'
// terms in FP64, four at a time in two chains.  The groups of the warp's
// species are one stream: the rates of the next group are on their way while
// a group is added.
struct Sums {
  const int4 *tm;
  int4 t0, t1, sg0;
  int s0, s1, list;
  __device__ __forceinline__ Sums(const FxTab &f, const unsigned char *tab, int list_, int gw)
      : list(list_) {
    s0 = reinterpret_cast<const int *>(tab + f.seg_ptr[list])[gw];
    s1 = reinterpret_cast<const int *>(tab + f.seg_ptr[list])[gw + 1];
    tm = reinterpret_cast<const int4 *>(tab + f.term[list]) +
         reinterpret_cast<const int *>(tab + f.term_ptr[list])[gw];
  }
  // the first terms, on their way before the barrier
  __device__ __forceinline__ void ahead(const FxTab &f, const unsigned char *tab) {
    t0 = __ldg(tm);
    t1 = __ldg(tm + 1);
    sg0 = __ldg(reinterpret_cast<const int4 *>(tab + f.seg[list]) + s0);
  }
  // q + col: the lane's column of the rates (a q that is the same for the
  // whole warp spares the scratch's 64-bit additions: 21.8 -> 20.9 ms, 2^22
  // states of 53/325); the state's sums to wdot if valid
  __device__ __forceinline__ void run(const FxTab &f, const unsigned char *tab,
                                      const unsigned char *q, unsigned col, double *wdot, int64_t ld,
                                      int64_t i, bool valid, int &bad) const {
    auto Q = [&](unsigned off) { return *reinterpret_cast<const double *>(q + off); };
    auto rates = [&](int4 t, double (&v)[4]) {
      const int x[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double d = Q(((unsigned)x[u] & 0x7fffff00u) | col);
        v[u] = __hiloint2double(__double2hiint(d) ^ (x[u] & 0x80000000), __double2loint(d));
      }
    };
    const int4 *tp = tm;
    double v[4];
    rates(t0, v);
    int4 t = t1, sgn = sg0;
#pragma unroll 1
    for (int a = s0; a < s1; ++a) {
      const int4 s = sgn;
      sgn = __ldg(reinterpret_cast<const int4 *>(tab + f.seg[list]) + a + 1);
      double w = 0.0, w2 = 0.0;
#pragma unroll 1
      for (int e = 0; e < s.y; ++e) {
        double u[4];
        rates(t, u);
        t = __ldg(tp + 2);
        ++tp;
        w += v[0];
        w2 += v[1];
        w += v[2];
        w2 += v[3];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = u[c];
      }
#pragma unroll 1
      for (int e = s.z; e < s.z + s.w; ++e)
        w = fma(__ldg(reinterpret_cast<const double *>(tab + f.wnu) + e),
                Q((unsigned)__ldg(reinterpret_cast<const int *>(tab + f.wterm) + e) | col), w);
      w += w2;
      if (valid) {
        bad += ((__double2hiint(w) >> 20) & 0x7ff) == 0x7ff;  // inf or NaN, integer test
        wdot[(int64_t)s.x * ld + i] = w;
      }
    }
  }
};

// Per-state values of a tile, one block of 32 states: rho, y_N, and the
// float-float T, ln T and 1/T, and P / (R T).
constexpr int BLOCK = 256 + 256 + 7 * 128;

// Sums, density and functions of T of one tile's states into the block at o,
// on warps 0-2, in the operations and the order of the one-state-per-thread
// kernel.  Called, not inlined: once per tile, and its registers are not the
// rate loops'.
__device__ __noinline__ void prepare(const Tab &t, const Batch &b, int64_t i, int warp, int lane,
                                     unsigned char *o) {
  double *rho = reinterpret_cast<double *>(o) + lane, *yN = rho + 32;
  const int N = t.N;
  const double *Y = b.Y + i;
  const int64_t ld = b.ld;
  if (warp == 0) {
    double ys = 0.0;
    int k = 0;
    for (; k + 8 <= N - 1; k += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = Y[(int64_t)(k + u) * ld];
#pragma unroll
      for (int u = 0; u < 8; ++u) ys += v[u];
    }
    for (; k < N - 1; ++k) ys += Y[(int64_t)k * ld];
    *yN = 1.0 - ys;
    asm volatile("bar.sync 1, 64;" ::: "memory");
  } else if (warp == 1) {
    double mwi = 0.0;
    int k = 0;
    for (; k + 8 <= N - 1; k += 8) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = Y[(int64_t)(k + u) * ld];
#pragma unroll
      for (int u = 0; u < 8; ++u) mwi = fma(v[u], t.inv_mw[k + u], mwi);
    }
    for (; k < N - 1; ++k) mwi = fma(Y[(int64_t)k * ld], t.inv_mw[k], mwi);
    asm volatile("bar.sync 1, 64;" ::: "memory");
    mwi = fma(*yN, t.inv_mw[N - 1], mwi);
    *rho = b.P[i] / mwi * ((1.0 / b.T[i]) * INV_RU);
  } else {
    const double T = b.T[i];
    const ff a = ff_from_double_int(T), l = ff_from_double_int(texp::log_t(T, t.logtab));
    const ff v = ff_from_double_int(1.0 / T);
    float *w = reinterpret_cast<float *>(o + 512) + lane;
    w[0] = a.h;
    w[32] = a.l;
    w[64] = l.h;
    w[96] = l.l;
    w[128] = v.h;
    w[160] = v.l;
    w[192] = d2f_rn(b.P[i] * (1.0 / T) * INV_RU);
  }
}

// The tile's concentrations, each as its mantissa in [1, 2) (zero: 0) and its
// binary exponent; row N: one, row N + 1: zero.
struct Conc {
  const unsigned char *p;
  __device__ __forceinline__ int2 at(unsigned off) const {
    return *reinterpret_cast<const int2 *>(p + off);
  }
  // (also inf and NaN; the subnormal are zero)
  __device__ __forceinline__ float operator[](int k) const {
    const int2 v = at(k * 256);
    return __int_as_float(v.x + (v.y << 23));
  }
};

// Stands in a rate's place until the general code has formed it: the loops
// that form the others then hold no call.
constexpr long long LATER = 0x7ff8c5a1d3b70e29ll;

// The warp's rates left to the general code, for the lane's state i:
// reactions without a record, exponents near or beyond the range of a double.
__device__ __noinline__ void finish(const unsigned char *img, const ImgLayout &lay,
                                    const unsigned char *src, int npairs, int n, const Batch &b,
                                    int64_t i, Conc C, const unsigned char *o, int lane,
                                    unsigned char *q, Scale *scale) {
  const Tab t = make_tab(img, lay);
  const float *w = reinterpret_cast<const float *>(o + 512) + lane;
  State s;
  s.T = b.T[i];
  s.P = b.P[i];
  s.invT = 1.0 / s.T;
  s.logT = texp::log_t(s.T, t.logtab);
  s.Tf = (float)s.T;
  s.Tff = ff{w[0], w[32]};
  s.lTff = ff{w[64], w[96]};
  s.iTff = ff{w[128], w[160]};
  KcMix kc;
  kc.Tbits = __double_as_longlong(s.T);
  kc.T = s.Tff;
  kc.logT = s.lTff;
  kc.invT = s.iTff;
  // the records: two for each pair, then one to a pair's place
#pragma unroll 1
  for (int p = 0; p < npairs + n; ++p) {
    const unsigned char *rec =
        src + (p < 2 * npairs ? (int64_t)p * MREC : (int64_t)(p - npairs) * MPAIR);
    const int r = __ldg(reinterpret_cast<const int *>(rec)) >> 8;
    double *v = reinterpret_cast<double *>(q + r * 256);
    if (__double_as_longlong(*v) != LATER) continue;
    double fwd, rev;
    float pm, sg;
    if (r >= t.R)
      *v = 0.0;
    else if (t.rate_kind[r] >= RATE_PLOG)
      *v = rxn_net<true>(t, r, s, w[192], C, kc, fwd, rev, pm);
    else if (const ff x = rate_exponent(t, r, s, sg); x.h != x.h)
      *v = __longlong_as_double(0x7ff8000000000000ll);
    else
      *v = rxn_net<false>(t, r, s, w[192], C, kc, fwd, rev, pm);
    if (scale) scale->add(*v);
  }
}

// A rate as it is formed: mantissa, its products' rounding errors, binary
// exponent + 896.
struct Rate {
  float m, err;
  int E;
  // exp(x) (ff_exp without its clamps: an x beyond them leaves E out of
  // range, as does NaN)
  __device__ __forceinline__ explicit Rate(ff x) {
    const float t = fmaf(x.h, LOG2E_F, SHIFT_F);
    const float kf = t - SHIFT_F;
    E = __float_as_int(t) - (0x4b400000 - 896);
    float r = fmaf(kf, -LN2_HI_F, x.h);
    r = fmaf(kf, -LN2_LO_F, r);
    r = r + x.l;
    float p = fmaf(r, 1.0f / 5040.0f, 1.0f / 720.0f);
    p = fmaf(p, r, 1.0f / 120.0f);
    p = fmaf(p, r, 1.0f / 24.0f);
    p = fmaf(p, r, 1.0f / 6.0f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    m = fmaf(p, r, 1.0f);
    err = 0.0f;
  }
  // FUSE: the last product may fuse with the addition of the errors, as in
  // the shape groups' code; else it is rounded by itself, as in product()
  template <bool FUSE>
  __device__ __forceinline__ void times(const Conc &C, unsigned off) {
    const int2 c = C.at(off);
    const float f = __int_as_float(c.x);
    const float mm = FUSE ? m * f : __fmul_rn(m, f);
    err = fmaf(err, f, fmaf(m, f, -mm));
    m = mm;
    E += c.y;
  }
  // (a mantissa between 2^-1 and 2^5, of a normal double with E in this range)
  __device__ __forceinline__ bool far() const { return (unsigned)(E + 120) > 2030u; }
  __device__ __forceinline__ double value(float sign = 1.0f) const {
    const float f = sign * (m + err);
    const unsigned u = __float_as_uint(f);
    const unsigned hi = ((u & 0x7fffffffu) >> 3) + ((unsigned)E << 20);
    return __hiloint2double((int)(f == 0.0f ? 0u : hi | (u & 0x80000000u)), (int)(u << 29));
  }
};
// offsets of the rows in the low and the high half of a word
__device__ __forceinline__ unsigned row_lo(int w) { return __byte_perm((unsigned)w, 0, 0x4104); }
__device__ __forceinline__ unsigned row_hi(int w) { return __byte_perm((unsigned)w, 0, 0x4324); }

// p * 2^k, rounded once, for a normal p and a result that may be subnormal or
// zero; |k| <= 250
__device__ __forceinline__ float scale2(float p, int k) {
  const int a = k >> 1;
  return p * __int_as_float((a + 127) << 23) * __int_as_float((k - a + 127) << 23);
}

// ff_expf, without calls
__device__ __forceinline__ float expf_of(ff x) {
  int k;
  const float p = ff_exp(x, k);
  const float v = scale2(p, min(max(k, -250), 250));
  return x.h > 88.0f ? INFINITY : x.h < -103.0f ? 0.0f : v;
}

// The fall-off factor of the record at r for a third-body concentration thd:
// mixed::pres_mod's operations without its calls and branches.
__device__ __forceinline__ float falloff(const unsigned char *r, int flags, float thd, ff T,
                                         ff lT, ff iT) {
  // ln k0 - ln kinf; every rounding as in the general code
  auto row = [&](int o, float &sign) {
    const float4 a = *reinterpret_cast<const float4 *>(r + o);
    const float4 c = *reinterpret_cast<const float4 *>(r + o + 16);
    sign = c.z;
    return ff_add(ff_add(ff{a.x, a.y}, ff_mul(ff{a.z, a.w}, lT)), ff_mul(ff{c.x, c.y}, iT));
  };
  float sign, none;
  const ff x0 = row(MFALL, sign), z = ff_add(x0, ff_neg(row(MFALL + 32, none)));
  int E, et, e2;
  float m = ff_exp(z, E);
  m = fsplit(m * fsplit(thd * sign, et), e2);
  E += et + e2;
  // Pr/(1+Pr) and 1/(1+Pr) from whichever of Pr and 1/Pr is at most 1
  const bool less = E < 0;
  const float s = scale2(less ? m : __frcp_rn(m), max(less ? E : -E, -250));
  const float d = __frcp_rn(1.0f + s), u = s * d;
  float frac = less ? u : d, inv1p = less ? d : u;
  if (m <= 0.0f) {
    frac = 0.0f;
    inv1p = 1.0f;
  }
  const float side = (flags & PMF_LOW) ? frac : inv1p;
  if (!(flags & (PMF_TROE | PMF_SRI))) return side;
  ff lnPr = ff{-1.0e30f, 0.0f};
  if (m > 0.0f) {
    const float Ef = (float)E;
    lnPr = ff_add(ff{Ef * LN2_H12_F, 0.0f}, ff{fmaf(Ef, LN2_L12_F, logf(m)), 0.0f});
  }
  ff lP = ff_mul(lnPr, ff{INV_LN10_F, INV_LN10_LO_F});
  if (lP.h < -300.0f) lP = ff{-300.0f, 0.0f};
  const float4 g = *reinterpret_cast<const float4 *>(r + MBROAD);
  const float4 h = *reinterpret_cast<const float4 *>(r + MBROAD + 16);
  // F = exp(ln base * w)
  float ln, F;
  ff w;
  if (flags & PMF_TROE) {
    // (the fused product is the one that the general code's compilation fuses)
    float f = fmaf(g.w, expf_of(ff_mul(T, ff{h.x, h.y})),
                   __fmul_rn(g.x, expf_of(ff_mul(T, ff{g.y, g.z}))));
    if (flags & PMF_T2) f += expf_of(ff_mul(iT, ff{h.z, h.w}));
    ln = logf(fmaxf(f, 1.0e-37f));
    const ff lF = ff_mul(ff{ln, 0.0f}, ff{INV_LN10_F, INV_LN10_LO_F});
    const ff A =
        ff_add(ff_add(lP, ff_neg(ff_mul(ff{0.6700000166893005f, -1.668930060816365e-08f}, lF))),
               ff{-0.4000000059604645f, 5.9604645663569045e-09f});
    const ff B =
        ff_add(ff_add(ff{0.8059999942779541f, 5.7220459481754915e-09f},
                      ff_neg(ff_mul(ff{1.176200032234192f, -3.2234190427971043e-08f}, lF))),
               ff_neg(ff_mul(ff{0.14000000059604645f, -5.9604643443123e-10f}, lP)));
    const ff B2 = ff_mul(B, B);
    w = ff_div(B2, ff_add(ff_mul(A, A), B2));
    F = expf_of(ff_mul(ff{ln, 0.0f}, w));
  } else {
    w = ff_div(ff{1.0f, 0.0f}, ff_add(ff{1.0f, 0.0f}, ff_mul(lP, lP)));
    ln = logf(g.x * expf_of(ff_mul(iT, ff{g.y, g.z})) + expf_of(ff_mul(T, ff{g.w, h.x})));
    F = expf_of(ff_mul(w, ff{ln, 0.0f}));
    if (flags & PMF_DE) F *= h.y * expf_of(ff_mul(ff{h.z, 0.0f}, lT));
  }
  return F * side;
}

// NW warps per CTA, CL CTAs (a cluster) per tile.  PACK: in place of the
// species sums, the contraction's operand -- each rate, scaled by the state's
// mean binary exponent, as bf16 hi and lo parts -- and the sums of the terms
// outside its window.  The operand is formed from the tile's rates while they
// are in L2.  Per 65,536 states of 561/2539: 3.04 ms; as kernels of their own
// with the rates through HBM, rates 3.92, operand 0.54, sums 0.83 ms.
template <int NW, int PER_SM, int CL, bool QS, bool PACK = false>
__global__ void __launch_bounds__(NW * 32, PER_SM)
    k_wdot_tile(const __grid_constant__ ImgLayout lay, const __grid_constant__ FxTab f,
                const __grid_constant__ Args g, const __grid_constant__ Batch b) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int N = f.N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned char *tab = g.tab;
  // shared memory: the concentrations [N + 2][32], 8 bytes each;
  // two blocks of per-state values; each warp's ring of records; the rates
  const Conc C{smem + lane * 8};
  unsigned char *next = smem + (N + 2) * 256;
  unsigned char *blk = next;
  next += 2 * BLOCK;
  unsigned char *ring = next + warp * (D * MPAIR);
  next += NW * (D * MPAIR);
  // (PACK) the warps' exponent sums, a bit per reaction with terms outside
  Scale *scales = reinterpret_cast<Scale *>(next) + threadIdx.x;
  unsigned *outside = reinterpret_cast<unsigned *>(next + NW * 32 * sizeof(Scale));
  __shared__ int s_slot;
  if (!QS && blockIdx.x % CL == 0 && threadIdx.x == 96)  // for the CTAs of the tile
    s_slot = tile::claim_slot(g.busy, g.slots, blockIdx.x / CL, b.status);
  unsigned char *qt = QS && CL > 1 ? static_cast<unsigned char *>(__cluster_map_shared_rank(next, 0))
                                   : next;  // (scratch: once there is a slot)
  unsigned char *q = qt + lane * 8;
  auto Q = [&](int off) -> double & { return *reinterpret_cast<double *>(q + off); };
  if (warp == 0) {
    int2 *c = reinterpret_cast<int2 *>(smem) + N * 32 + lane;
    c[0] = make_int2(0x3f800000, 0);
    c[32] = make_int2(0, 0);
    if (QS) reinterpret_cast<double *>(next)[f.R * 32 + lane] = 0.0;  // before all CTAs run
  }
  const int gw = CL == 1 ? warp : (int)(blockIdx.x % CL) * NW + warp;  // the tile's warp
  const int *lp = reinterpret_cast<const int *>(tab + f.mlist_ptr[g.list]) + gw;
  const Ring<D> recs{tab + f.mrec[g.list] + (int64_t)lp[0] * MPAIR, smem_u32(ring), MPAIR,
                     lp[1] - lp[0], lane};
  const int npairs = reinterpret_cast<const int *>(tab + f.mpairs[g.list])[gw];
  int bad = 0, bk = 0;
  int64_t tile = blockIdx.x / CL;
  const int64_t step = gridDim.x / CL;
  const int64_t ntiles = (b.n + 31) / 32;
  const Tab t = make_tab(g.img, lay);
  if (tile < ntiles && warp < 3)
    prepare(t, b, tile * 32 + lane < b.n ? tile * 32 + lane : tile * 32, warp, lane, blk);
  if (!QS) {  // (the claim ran beside the first tile's sums)
    tile_barrier<CL>();
    int slot = CL > 1 ? *static_cast<const int *>(__cluster_map_shared_rank(&s_slot, 0)) : s_slot;
    // the same for the whole warp, and known to be (see Sums::run: 2^18 states of
    // 53/325 1.39 -> 1.35 ms)
    if (!PACK) slot = __shfl_sync(0xffffffffu, slot, 0);
    qt = reinterpret_cast<unsigned char *>(g.q) + (int64_t)slot * (f.R + 1) * 256;
    q = qt + lane * 8;
    if (warp == 0) Q(f.R * 256) = 0.0;
  }
  Sums sums(f, tab, g.list, gw);
  for (; tile < ntiles; tile += step, bk ^= 1) {
    const int64_t i = tile * 32 + lane;
    const bool valid = i < b.n;
    const int64_t ic = valid ? i : tile * 32;  // idle lanes repeat a valid state
    tile_barrier<CL>();
    recs.start();
    if (PACK)
      for (int k = threadIdx.x; k <= f.R / 32; k += NW * 32) outside[k] = 0;
    const unsigned char *o = blk + bk * BLOCK;
    const double rho = reinterpret_cast<const double *>(o)[lane];
#pragma unroll 4
    for (int k = warp; k < N; k += NW) {
      const double y = k == N - 1 ? reinterpret_cast<const double *>(o + 256)[lane]
                                  : b.Y[(int64_t)k * b.ld + ic];
      int2 c;
      c.x = __float_as_int(fsplit(d2f_rn(y * (rho * __ldg(t.inv_mw + k))), c.y));
      reinterpret_cast<int2 *>(smem)[k * 32 + lane] = c;
    }
    __syncthreads();
    // net rates
    if (warp < 3 && tile + step < ntiles) {
      const int64_t j = (tile + step) * 32;
      prepare(t, b, j + lane < b.n ? j + lane : j, warp, lane, blk + (bk ^ 1) * BLOCK);
    }
    {
      const float *w = reinterpret_cast<const float *>(o + 512) + lane;
      const ff T{w[0], w[32]}, lT{w[64], w[96]}, iT{w[128], w[160]};
      const long long Tbits = __double_as_longlong(b.T[ic]);
      auto forward = [&](const unsigned char *r) {
        const float4 a = *reinterpret_cast<const float4 *>(r + 16);
        const float2 c = *reinterpret_cast<const float2 *>(r + 32);
        ff v = ff_fma(ff{a.z, a.w}, lT, ff{a.x, a.y});
        v = ff_fma(ff{c.x, c.y}, iT, v);
        return ff_norm(v.h, v.l);
      };
      // forward minus Kc, from its own coefficients
      auto reverse = [&](const unsigned char *r) {
        const longlong2 *lo3 = reinterpret_cast<const longlong2 *>(r + 96);
        const float4 *c = reinterpret_cast<const float4 *>(r + 48 + (Tbits <= lo3->y ? 0 : 64));
        const float4 a = c[0], d = c[1], e = c[2], h = c[3];
        ff v = ff{e.z, e.w};
        v = ff_fma(v, T, ff{e.x, e.y});
        v = ff_fma(v, T, ff{d.z, d.w});
        v = ff_fma(v, T, ff{d.x, d.y});
        v = ff_fma(v, T, ff{a.x, a.y});
        v = ff_fma(ff{a.z, a.w}, lT, v);
        v = ff_fma(ff{h.x, h.y}, iT, v);
        return ff_norm(v.h, v.l);
      };
      int slot = 0;
      bool later = false;
      Scale scale;
      auto put = [&](int off, double v) {
        Q(off) = v;
        if (PACK) scale.add(v);
      };
#pragma unroll 1
      for (int p = 0; p < npairs; ++p) {
        const unsigned char *at = ring + slot * MPAIR;
        slot = recs.next(p, slot);
        const int4 h0 = *reinterpret_cast<const int4 *>(at);
        const int4 h1 = *reinterpret_cast<const int4 *>(at + MREC);
        const bool more = h0.x & MF_MORE;
        Rate f0(forward(at)), f1(forward(at + MREC));
        f0.times<true>(C, row_lo(h0.y));
        f1.times<true>(C, row_lo(h1.y));
        f0.times<true>(C, row_hi(h0.y));
        f1.times<true>(C, row_hi(h1.y));
        if (more) {
          f0.times<true>(C, row_lo(h0.z));
          f1.times<true>(C, row_lo(h1.z));
        }
        bool far = f0.far() || f1.far();
        double v0 = f0.value(), v1 = f1.value();
        if (h0.x & MF_REV) {
          Rate r0(reverse(at)), r1(reverse(at + MREC));
          r0.times<true>(C, row_hi(h0.z));
          r1.times<true>(C, row_hi(h1.z));
          r0.times<true>(C, row_lo(h0.w));
          r1.times<true>(C, row_lo(h1.w));
          if (more) {
            r0.times<true>(C, row_hi(h0.w));
            r1.times<true>(C, row_hi(h1.w));
          }
          far |= r0.far() || r1.far();
          v0 -= r0.value();  // FP64
          v1 -= r1.value();
        }
        if (far) v0 = v1 = __longlong_as_double(LATER);
        later |= far;
        put(h0.x & ~255, v0);
        put(h1.x, v1);
      }
#pragma unroll 1
      for (int p = npairs; p < recs.n; ++p) {
        const unsigned char *at = ring + slot * MPAIR;
        slot = recs.next(p, slot);
        const int4 h = *reinterpret_cast<const int4 *>(at);
        bool far = h.x & MF_GEN;
        double v = 0.0;
        if (!far) {
          float pm = 0.0f;
          if (h.x & (MF_THD | MF_FALL)) {
            const int4 ph = *reinterpret_cast<const int4 *>(at + MPM);
            if (ph.w >= 0) {
              pm = C[ph.w];
            } else {
              pm = reinterpret_cast<const float *>(o + 512 + 768)[lane];
              const float4 *e = reinterpret_cast<const float4 *>(at + MEFFS);
#pragma unroll 1
              for (int c = 0; c < ph.x; c += 2) {
                if (c == MEFF) e = reinterpret_cast<const float4 *>(tab + ph.y) - MEFF / 2;
                const float4 w = e[c / 2];
                pm = fmaf(w.x, C[__float_as_int(w.y)], pm);
                pm = fmaf(w.z, C[__float_as_int(w.w)], pm);
              }
            }
            if (h.x & MF_FALL) pm = falloff(at, ph.z, pm, T, lT, iT);
          }
          const float sg = *reinterpret_cast<const float *>(at + 40);
          Rate f(forward(at)), r(reverse(at));
          f.times<false>(C, row_lo(h.y));
          r.times<false>(C, row_hi(h.z));
          f.times<false>(C, row_hi(h.y));
          r.times<false>(C, row_lo(h.w));
          f.times<false>(C, row_lo(h.z));
          r.times<false>(C, row_hi(h.w));
          v = f.value(sg);
          far = f.far();
          if (h.x & MF_REV) {
            v -= r.value(sg);  // FP64
            far |= r.far();
          }
          if (h.x & (MF_THD | MF_FALL)) v *= f2d_exact(pm);
        }
        if (far) v = __longlong_as_double(LATER);
        later |= far;
        put(h.x & ~255, v);
      }
      if (PACK) *scales = scale;
      if (later)
        finish(g.img, lay, recs.src, npairs, recs.n, b, ic, C, o, lane, q,
               PACK ? scales : nullptr);
    }
    if constexpr (PACK) {
      __syncthreads();
      int es = 0, ec = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const Scale a = scales[(w - warp) * 32];
        es += a.sum;
        ec += a.count;
      }
      const int c = tile::scale_exponent(es, ec);
      if (warp == 0 && valid) g.escale[i] = c;
      __nv_bfloat16 *row = g.A + i * (2 * (int64_t)g.Kh);
#pragma unroll 1
      for (int r0 = warp * 16; r0 < g.Kh; r0 += NW * 16) {
        unsigned hi[8], lo[8];
#pragma unroll
        for (int u = 0; u < 16; u += 2) {
          float x[2];
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int r = r0 + u + w;
            const double v = r < f.R ? Q(r * 256) : 0.0;
            const bool in = in_window(v, c);
            if (__any_sync(0xffffffffu, valid && !in) && lane == 0)
              atomicOr(&outside[r >> 5], 1u << (r & 31));
            // v * 2^-c exactly through the exponent field (the result stays a
            // normal number within 2^+-WINDOW), then rounded to fp32
            x[w] = in && v != 0.0 ? d2f_rn(__hiloint2double(__double2hiint(v) - c * (1 << 20),
                                                            __double2loint(v)))
                                  : 0.0f;
          }
          const __nv_bfloat162 h = __floats2bfloat162_rn(x[0], x[1]);
          const __nv_bfloat162 l = __floats2bfloat162_rn(x[0] - __low2float(h),
                                                         x[1] - __high2float(h));
          hi[u / 2] = *reinterpret_cast<const unsigned *>(&h);
          lo[u / 2] = *reinterpret_cast<const unsigned *>(&l);
        }
        if (valid) {
          store32(row + r0, hi);
          store32(row + g.Kh + r0, lo);
        }
      }
      __syncthreads();
      // terms outside the window in FP64, in reaction order per species; 32
      // terms are looked up at a time
#pragma unroll 1
      for (int k = warp; k < N; k += NW) {
        double w = 0.0;
        const int e1 = __ldg(t.spc_ptr + k + 1);
#pragma unroll 1
        for (int e = __ldg(t.spc_ptr + k); e < e1; e += 32) {
          const int r = e + lane < e1 ? __ldg(t.spc_r + e + lane) : -1;
          unsigned some =
              __ballot_sync(0xffffffffu, r >= 0 && (outside[r >> 5] >> (r & 31) & 1u));
          for (; some; some &= some - 1) {
            const int j = __ffs(some) - 1;
            const double v = Q(__shfl_sync(0xffffffffu, r, j) * 256);
            if (!in_window(v, c)) w = fma(__ldg(t.spc_nu + e + j), v, w);
          }
        }
        if (valid) b.wdot[(int64_t)k * b.ld + i] = w;
      }
      continue;  // rates and bits are replaced after the barrier at the loop's head
    }
    sums.ahead(f, tab);
    tile_barrier<CL>();
    sums.run(f, tab, qt, (unsigned)lane * 8, b.wdot, b.ld, i, valid, bad);
    // rates are replaced only after the barrier at the loop's head
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (!QS || CL > 1) tile_barrier<CL>();  // the tile's rates are read until here
  if (!QS && blockIdx.x % CL == 0 && threadIdx.x == 0)
    tile::release_slot(g.busy, g.slots, s_slot);
  if (bad && b.status) atomicAdd(&b.status[1], bad);
}

size_t smem_of(const FxTab &f, int nw, bool qs, bool pack = false) {
  return (pack ? (size_t)nw * 32 * sizeof(Scale) + (f.R / 32 + 1) * 4 : 0) +
         (size_t)(f.N + 2) * 256 + 2 * BLOCK + (size_t)nw * D * MPAIR +
         (qs ? (size_t)(f.R + 1) * 256 : 0);
}

struct Plan {
  int nw = 24, per_sm = 1, cl = 1;
  bool qs = false, ok = false;
};

Plan plan_of(const FxTab &f, int64_t tiles, int sm_count, int smem_optin) {
  if (!f.mixed) return Plan{};
  // the lines of crs_fx.cu, whose shapes these are: 1,024 states of 53/325
  // (clusters) 28.7 us, 5,000 (three CTAs per SM) 72 us; one state per thread
  // took 455 us for either
  auto fits = [&](int nw, int per_sm, bool qs) {
    return (smem_of(f, nw, qs) + 1024) * per_sm <= (size_t)smem_optin + 1024;
  };
  for (int cl = 8; cl > 1; cl /= 2)
    if (tiles * cl <= sm_count && f.R >= 32 * cl) {
      if (fits(16, 1, true)) return Plan{16, 1, cl, true, true};
      if (fits(16, 1, false)) return Plan{16, 1, cl, false, true};
    }
  if (tiles <= sm_count && fits(16, 1, true)) return Plan{16, 1, 1, true, true};
  if (f.R < 100 && fits(4, 6, true)) return Plan{4, 6, 1, true, true};
  if (fits(8, 3, false)) return Plan{8, 3, 1, false, true};
  Plan p{24, 1, 1, false, false};
  p.ok = fits(24, 1, false);
  return p;
}

using Kernel = void (*)(const ImgLayout, const FxTab, const Args, const Batch);
Kernel kernel_of(const Plan &p) {
  switch (p.cl) {
    case 8: return p.qs ? k_wdot_tile<16, 1, 8, true> : k_wdot_tile<16, 1, 8, false>;
    case 4: return p.qs ? k_wdot_tile<16, 1, 4, true> : k_wdot_tile<16, 1, 4, false>;
    case 2: return p.qs ? k_wdot_tile<16, 1, 2, true> : k_wdot_tile<16, 1, 2, false>;
  }
  if (p.nw == 4) return k_wdot_tile<4, 6, 1, true>;
  if (p.nw == 16) return k_wdot_tile<16, 1, 1, true>;
  if (p.nw == 8) return k_wdot_tile<8, 3, 1, false>;
  return k_wdot_tile<24, 1, 1, false>;
}

// the contraction's producer: one CTA of 24 warps per SM
constexpr int PACK_NW = 24;
constexpr Kernel k_pack = k_wdot_tile<PACK_NW, 1, 1, false, true>;

}  // namespace mixt

cudaError_t mixed_tile_init(int smem_optin) {
  cudaError_t e = cudaSuccess;
  e = set_smem_limit(mixt::k_pack, (size_t)smem_optin);
  for (int q = 0; q < 7 && e == cudaSuccess; ++q) {
    mixt::Plan p;
    p.cl = q < 3 ? 2 << q : 1;
    p.nw = q == 3 ? 4 : q == 4 ? 16 : q == 5 ? 8 : 24;
    p.qs = true;
    e = set_smem_limit(mixt::kernel_of(p), (size_t)smem_optin);
    p.qs = false;
    if (e == cudaSuccess) e = set_smem_limit(mixt::kernel_of(p), (size_t)smem_optin);
  }
  return e;
}

// Whether the contraction's producer takes the mechanism (it needs scratch).
bool mixed_pack_fits(const fx::FxTab &f, int smem_optin) {
  return f.mixed && mixt::smem_of(f, mixt::PACK_NW, false, true) <= (size_t)smem_optin;
}

static int64_t mixed_first(const fx::FxTab &f, int64_t tiles, int sm_count, int smem_optin) {
  const mixt::Plan p = mixt::plan_of(f, tiles, sm_count, smem_optin);
  const int64_t wave = (int64_t)sm_count * p.per_sm;
  const int64_t rest = tiles % wave;
  return p.cl > 1 || tiles < wave || rest == 0 || 2 * rest > sm_count || f.R < 64 ? tiles
                                                                                  : tiles - rest;
}

int mixed_tile_scratch(const fx::FxTab &f, int64_t n, int sm_count, int smem_optin) {
  const int64_t tiles = (n + 31) / 32, first = mixed_first(f, tiles, sm_count, smem_optin);
  int need = 0;
  for (int64_t part : {first, tiles - first}) {
    if (part == 0) continue;
    const mixt::Plan p = mixt::plan_of(f, part, sm_count, smem_optin);
    if (!p.ok) return -1;
    need |= !p.qs;
  }
  return need;
}

// The resources of the launches that need scratch.
cudaError_t mixed_tile_slots(const fx::FxTab &f, int sm_count, int smem_optin, SlotUse &u) {
  cudaError_t e = cudaSuccess;
  for (int64_t tiles : {1, sm_count / 8 + 1, sm_count / 4 + 1, sm_count / 2 + 1, sm_count + 1}) {
    const mixt::Plan p = mixt::plan_of(f, tiles, sm_count, smem_optin);
    if (p.ok && !p.qs && e == cudaSuccess)
      e = u.add(mixt::kernel_of(p), p.nw * 32, mixt::smem_of(f, p.nw, p.qs));
  }
  if (e == cudaSuccess && mixed_pack_fits(f, smem_optin))
    e = u.add(mixt::k_pack, mixt::PACK_NW * 32, mixt::smem_of(f, mixt::PACK_NW, false, true));
  return e;
}

static cudaError_t launch_mixed_part(const unsigned char *img, const ImgLayout &L,
                                     const fx::FxTab &f, const unsigned char *tab, const Batch &b,
                                     int sm_count, int smem_optin, const TileScratch &scratch,
                                     cudaStream_t s) {
  const int64_t tiles = (b.n + 31) / 32;
  const mixt::Plan p = mixt::plan_of(f, tiles, sm_count, smem_optin);
  if (!p.ok || (!p.qs && !scratch.q)) return cudaErrorInvalidValue;
  int list = 0;
  while (list < fx::NLIST - 1 && fx::list_warps[list] != p.nw * p.cl) ++list;
  const mixt::Kernel k = mixt::kernel_of(p);
  const size_t bytes = mixt::smem_of(f, p.nw, p.qs);
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
  const mixt::Args args{tab, img, scratch.q, scratch.busy, scratch.slots, list, nullptr, 0, nullptr};
  return cudaLaunchKernelEx(&cfg, k, L, f, args, b);
}

cudaError_t launch_mixed_tile(const unsigned char *img, const ImgLayout &L, const fx::FxTab &f,
                              const unsigned char *tab, const Batch &b, int sm_count,
                              int smem_optin, const TileScratch &scratch, cudaStream_t s) {
  const int64_t tiles = (b.n + 31) / 32, first = mixed_first(f, tiles, sm_count, smem_optin);
  Batch part = b;
  part.n = std::min<int64_t>(b.n, first * 32);
  cudaError_t e = launch_mixed_part(img, L, f, tab, part, sm_count, smem_optin, scratch, s);
  if (e != cudaSuccess || first == tiles) return e;
  const int64_t o = part.n;
  part.n = b.n - o;
  part.T += o;
  part.P += o;
  part.Y += o;
  part.wdot += o;
  return launch_mixed_part(img, L, f, tab, part, sm_count, smem_optin, scratch, s);
}

// A: rows of 2 Kh (a multiple of 64), 32-byte aligned.
cudaError_t launch_mixed_pack(const unsigned char *img, const ImgLayout &L, const fx::FxTab &f,
                              const unsigned char *tab, const Batch &b, int sm_count,
                              int smem_optin, const TileScratch &scratch, void *A, int Kh,
                              int *escale, cudaStream_t s) {
  if (!mixed_pack_fits(f, smem_optin) || !scratch.q || Kh % 64 || Kh < f.R)
    return cudaErrorInvalidValue;
  int list = 0;
  while (list < fx::NLIST - 1 && fx::list_warps[list] != mixt::PACK_NW) ++list;
  mixt::k_pack<<<(unsigned)std::min<int64_t>((b.n + 31) / 32, sm_count), mixt::PACK_NW * 32,
                 mixt::smem_of(f, mixt::PACK_NW, false, true), s>>>(
      L, f,
      mixt::Args{tab, img, scratch.q, scratch.busy, scratch.slots, list,
                 static_cast<__nv_bfloat16 *>(A), Kh, escale},
      b);
  return cudaGetLastError();
}

}  // namespace crs
