// Pieces that the state-tile kernels share (crs_fx.cu, crs_mixed_tile.cu): a
// warp's ring of reaction records in shared memory, the barrier of the CTAs
// of a tile, and the species sums over a tile's net rates.
#pragma once

#include "crs_fx_tab.cuh"
#include "crs_internal.cuh"

namespace crs {
namespace fx {

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
  // whole warp spares the scratch's 64-bit additions: 21.8 -> 20.9 ms for
  // mixed precision, 2^22 states of 53/325; in the FP64 kernel, with its own
  // registers, 6.42 -> 6.56 ms for 2^20); the state's sums to wdot if valid
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

}  // namespace fx
}  // namespace crs
