// Tables of the FP64 state-tile kernel (crs_fx.cu), in a device buffer of
// their own beside the mechanism's table image.
#pragma once

#include <cstdint>
#include <vector>

#include "../../include/crs_tables.h"

namespace crs {
namespace fx {

// Temperature intervals (tb[q], tb[q + 1]] on which the functions of T are
// normalised; the second bound is the mechanism's most common T_common.
constexpr int NI = 2;
// Work lists for so many warps per tile (a CTA's, or a cluster's).
constexpr int NLIST = 7;
constexpr int list_warps[NLIST] = {4, 8, 16, 24, 32, 64, 128};
// A reaction's record: its head, int4 {slot offset, flags, fall-off entry,
// reaction}, int4 {two reactants, two products}, int4 {the third and fourth
// of each}, as offsets of tile rows; for reactions with pressure
// modification int4 {flags, species row or -1, 0, 0} and a record per
// interval; its coefficients per interval; its T thresholds if any.
constexpr int HEAD = 48;
constexpr int PMH = 16, PMC = 96;
constexpr int COEF = 80;
constexpr int BASIS = 9;  // words of an interval's normalisation

// reaction flags (RF_NEG is bit 0: the sign bit of an exponent)
enum { RF_NEG = 1, RF_REV = 2, RF_THD = 4, RF_FALL = 8, RF_GEN = 16, RF_MORE = 32 };
// pressure-modification flags; T1, T2, T3: exponential terms present
enum { PMF_LOW = 1, PMF_TROE = 2, PMF_SRI = 4, PMF_DE = 8, PMF_T1 = 16, PMF_T2 = 32,
       PMF_T3 = 64 };

// Passed by value; offsets in bytes into the buffer.
struct FxTab {
  int N, R, NPM;
  int usable;            // the kernel takes this mechanism
  int nthr;              // T thresholds per reaction record; 0: the interval bounds
  int stride[2];         // bytes of a pair of plain reversible reactions' records and of
                         // another reaction's
  double tb[NI + 1];
  int small, hp, basis;  // exponential and logarithm tables; log2 T; normalisation
  int lw;                // [N] log2(1 / W_k)
  int pm;                // [NPM] int2 {slot offset or -1: no third-body sum, 0}
  int eff_ptr, eff;      // third-body lists: {double (eff - 1) / W, int row offset, int 0}
  // per warp: its plain reversible reactions' records in pairs (an odd
  // number is completed with one that puts zero into the slot of zeros), its
  // other reactions' records, and its species' terms
  int list_ptr[NLIST][2], rec[NLIST][2];
  // its species, int4 {species, groups of terms, first weighted term, their
  // number}, those with weighted terms last; its groups of four terms {slot
  // offset, bit 31: subtract}, one after another, completed with the slot of
  // zeros (row R)
  int seg_ptr[NLIST], seg[NLIST], term_ptr[NLIST], term[NLIST];
  int wterm, wnu;
  // mixed precision (crs_mixed_tile.cu), in the same lists: per warp, its
  // records (lists of MPAIR bytes each), those of pairs of shape-group
  // reactions first
  int mixed;  // the kernel takes this mechanism
  int mlist_ptr[NLIST], mpairs[NLIST], mrec[NLIST];
  int bytes;
};
// A mixed record: int {slot offset | MF flags}, uint16 {three reactants, three
// products} as rows of the tile, the rate row, the Kc polynomials.  Two of
// them are a pair; a reaction outside the shape groups has one, then int4
// {third-body terms, the first beyond the record, PMF flags, species row},
// the fall-off's two rate rows, its broadening's coefficients and MEFF
// third-body terms {float, int row}.
constexpr int MREC = 16 + 32 + 128, MPAIR = 2 * MREC;
constexpr int MPM = MREC, MFALL = MPM + 16, MBROAD = MFALL + 64, MEFFS = MBROAD + 32;
constexpr int MEFF = (MPAIR - MEFFS) / 8;
// (of a pair's first record: some factor is a third one; reversible)
enum { MF_MORE = 1, MF_REV = 2, MF_THD = 4, MF_FALL = 8, MF_GEN = 16 };

// The tables of a mechanism; none (f.usable = f.mixed = 0) when they might
// take more than `limit` bytes or more than 32-bit offsets reach, from some
// 390,000 reactions on.
void build(const Tab &t, FxTab &f, std::vector<unsigned char> &out, int64_t limit = INT32_MAX);

}  // namespace fx
}  // namespace crs
