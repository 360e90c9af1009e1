// Tables of the FP64 state-tile kernel (crs_fx.cu), in a device buffer of
// their own beside the mechanism's table image.
#pragma once

#include <cstdint>

namespace crs {
namespace fx {

// Temperature intervals (TB[q], TB[q + 1]] on which the functions of T are
// normalised; the middle bound is the mechanism's most common T_common.
constexpr int NI = 3;
constexpr int NLIST = 3;               // work lists for 4, 8 and 16 warps per CTA
constexpr int COEF = 10;               // 8-byte words per coefficient record
constexpr int PMC = 12;                // and per pressure-modification record
constexpr int BASIS = 9;               // and per interval's normalisation

// reaction flags
enum { RF_REV = 1, RF_THD = 2, RF_FALL = 4, RF_GEN = 8, RF_MORE_R = 16, RF_MORE_P = 32,
       RF_NEG = 64 };
// pressure-modification flags; T1, T2, T3: exponential terms present
enum { PMF_LOW = 1, PMF_TROE = 2, PMF_SRI = 4, PMF_DE = 8, PMF_T1 = 16, PMF_T2 = 32,
       PMF_T3 = 64, PMF_SUM = 128 };

// Passed by value; offsets in bytes into the buffer.
struct FxTab {
  int N, R, NPM;
  int usable;       // the kernel takes this mechanism
  int uniform;      // every reaction changes coefficients at the interval bounds only
  int eff_shift;    // third-body sums are formed in units of 2^eff_shift
  double tb[NI + 1];
  int small, hp, basis;        // exponential and logarithm tables; log2 T; normalisation
  int lw;                      // [N] log2(1 / W_k)
  int hdr, coef;               // [R] 2 x int4; coefficient records
  int thr_ptr, thr;            // [R + 1], T thresholds of each reaction (uniform = 0)
  int pmh, pmc;                // [NPM] int4 {flags, species, reaction, 0}; [NPM][NI] records
  int eff_ptr, eff_sp, eff_k;  // third-body lists
  // per warp: its reactions, plain reversible ones first (their number in
  // list_rev), and its species
  int list_ptr[NLIST], list_rev[NLIST], list[NLIST];
  int sum_ptr[NLIST], sum[NLIST];
  int bytes;
};

constexpr int warps_of(int list) { return 4 << list; }

}  // namespace fx
}  // namespace crs
