// Surrogate network kernels: a BF16 MLP trained and evaluated on the
// tensor cores.
//
// Layers are Y = act(X W^T + b) computed by the tcgen05 GEMM of
// crs_gemm.cuh with fused epilogues:
//   forward          z = acc + b; a = silu(z); store z (fp32, for the
//                    backward pass), a row-major (bf16, the next layer's X)
//                    and a transposed (bf16, the operand of the weight
//                    gradient), or the fp32 output of the last layer;
//   backward, data   dz_prev = (dz W) * silu'(z_prev), stored row-major and
//                    transposed (bf16);
//   backward, weight dW = dz^T a_prev, split over K (the batch) into fp32
//                    partial sums reduced in a fixed order.
// Element-wise kernels: input features and the training-set box check,
// loss and its gradient, bias gradients, Adam (fp32 master weights, bf16
// copies W and W^T), and the surrogate's output transform with the
// element-conservation check that routes states back to the exact kernel.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>

#include "../../include/crs.h"
#include "crs_gemm.cuh"
#include "crs_internal.cuh"

namespace crs {
namespace mlp {

__device__ __forceinline__ float sigmoidf(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoidf(z); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = sigmoidf(z);
  return s * (1.0f + z * (1.0f - s));
}

// Stores of one thread's 32 consecutive values of a row: four or eight
// 16-byte stores when all 32 are wanted and the address allows it (rows of
// a warp are a row stride apart, so per-element stores would cost a memory
// sector each), element by element otherwise.
__device__ __forceinline__ void store32(float *dst, const float (&x)[32], int nvalid) {
  if (nvalid >= 32 && !(reinterpret_cast<uintptr_t>(dst) & 15)) {
    float4 *d = reinterpret_cast<float4 *>(dst);
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < nvalid) dst[j] = x[j];
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void store32(__nv_bfloat16 *dst, const float (&x)[32], int nvalid) {
  if (nvalid >= 32 && !(reinterpret_cast<uintptr_t>(dst) & 15)) {
    uint4 *d = reinterpret_cast<uint4 *>(dst);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      d[q] = make_uint4(pack_bf16(x[8 * q], x[8 * q + 1]), pack_bf16(x[8 * q + 2], x[8 * q + 3]),
                        pack_bf16(x[8 * q + 4], x[8 * q + 5]),
                        pack_bf16(x[8 * q + 6], x[8 * q + 7]));
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < nvalid) dst[j] = __float2bfloat16_rn(x[j]);
  }
}

struct EpiForward {
  const float *bias;  // [N] or nullptr
  int act;
  int m_valid, n_valid;
  float *Z;
  int64_t ldz;
  __nv_bfloat16 *A;
  int64_t lda;
  __nv_bfloat16 *AT;
  int64_t ldat;
  float *Y;
  int64_t ldy;
  __device__ void operator()(int row, int col0, const uint32_t (&v)[32]) const {
    if (row >= m_valid || col0 >= n_valid) return;
    const int nv = n_valid - col0;
    float z[32], a[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      z[j] = __uint_as_float(v[j]) + ((bias && j < nv) ? bias[col0 + j] : 0.0f);
      a[j] = act == CRS_ACT_SILU ? silu(z[j]) : z[j];
    }
    if (Z) store32(Z + (int64_t)row * ldz + col0, z, nv);
    if (A) store32(A + (int64_t)row * lda + col0, a, nv);
    if (Y) store32(Y + (int64_t)row * ldy + col0, a, nv);
    if (AT) {
      // consecutive lanes hold consecutive rows: these stores coalesce
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < nv) AT[(int64_t)(col0 + j) * ldat + row] = __float2bfloat16_rn(a[j]);
    }
  }
};

struct EpiBackwardData {
  const float *Zprev;
  int64_t ldz;
  int m_valid, n_valid;
  __nv_bfloat16 *dZ;
  int64_t ld;
  __nv_bfloat16 *dZT;
  int64_t ldt;
  __device__ void operator()(int row, int col0, const uint32_t (&v)[32]) const {
    if (row >= m_valid || col0 >= n_valid) return;
    const int nv = n_valid - col0;
    const float *zp = Zprev + (int64_t)row * ldz + col0;
    float zv[32], d[32];
    if (nv >= 32 && !(reinterpret_cast<uintptr_t>(zp) & 15)) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 t = reinterpret_cast<const float4 *>(zp)[q];
        zv[4 * q] = t.x;
        zv[4 * q + 1] = t.y;
        zv[4 * q + 2] = t.z;
        zv[4 * q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) zv[j] = j < nv ? zp[j] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) d[j] = __uint_as_float(v[j]) * dsilu(zv[j]);
    store32(dZ + (int64_t)row * ld + col0, d, nv);
    if (dZT) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < nv) dZT[(int64_t)(col0 + j) * ldt + row] = __float2bfloat16_rn(d[j]);
    }
  }
};

// split-K partial: P[z][row][col]
struct EpiPartial {
  float *P;
  int64_t rows_pad, cols_pad;
  __device__ void operator()(int row, int col0, const uint32_t (&v)[32]) const {
    float x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
    store32(P + ((int64_t)blockIdx.z * rows_pad + row) * cols_pad + col0, x, 32);
  }
};

// Sums in slice order, eight slices of loads in flight.
__global__ void __launch_bounds__(256)
    k_reduce_partials(const float *P, int splits, int64_t rows_pad, int64_t cols_pad,
                      int64_t rows, int64_t cols, float *dW) {
  const int64_t n = rows * cols, slice = rows_pad * cols_pad;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const float *p = P + idx / cols * cols_pad + idx % cols;
    float s = 0.0f;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) s += p[z * slice];
    dW[idx] = s;
  }
}

// Row sums of a [rows][ld] bf16 matrix over its first m columns, a warp per row
// with a column per lane: short rows, and rows enough to fill the chip.
__global__ void __launch_bounds__(256)
    k_row_sums_short(const __nv_bfloat16 *X, int64_t ld, int64_t rows, int64_t m, float *out) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  float s = 0.0f;
  for (int64_t i = lane; i < m; i += 32) s += __bfloat162float(X[row * ld + i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[row] = s;
}

// The same sums of few long rows: a CTA per row.  The order of summation is
// that of a warp per row, whose 2-byte
// loads took 30 us for 256 rows of 16,384: here seven warps bring the next
// 4,096 columns on chip, eight per load where the row's address allows it,
// while the first adds the present ones.
constexpr int ROW_CHUNK = 4096;
__global__ void __launch_bounds__(256)
    k_row_sums(const __nv_bfloat16 *X, int64_t ld, int64_t m, float *out) {
  __shared__ __align__(16) __nv_bfloat16 buf[2][ROW_CHUNK];
  const __nv_bfloat16 *x = X + (int64_t)blockIdx.x * ld;
  const bool quads = !(reinterpret_cast<uintptr_t>(x) & 15);
  const int lane = threadIdx.x & 31;
  auto fetch = [&](int64_t c0, __nv_bfloat16 *to) {
    const int cnt = m - c0 < ROW_CHUNK ? (int)(m - c0) : ROW_CHUNK;
    const int done = quads ? cnt / 8 * 8 : 0;
    for (int i = ((int)threadIdx.x - 32) * 8; i < done; i += 224 * 8)
      *reinterpret_cast<uint4 *>(to + i) = *reinterpret_cast<const uint4 *>(x + c0 + i);
    for (int i = done + (int)threadIdx.x - 32; i < cnt; i += 224) to[i] = x[c0 + i];
  };
  if (threadIdx.x >= 32) fetch(0, buf[0]);
  float s = 0.0f;
  for (int64_t c0 = 0, k = 0; c0 < m; c0 += ROW_CHUNK, ++k) {
    __syncthreads();
    if (threadIdx.x >= 32) {
      if (c0 + ROW_CHUNK < m) fetch(c0 + ROW_CHUNK, buf[(k + 1) & 1]);
    } else {
      const int cnt = m - c0 < ROW_CHUNK ? (int)(m - c0) : ROW_CHUNK;
#pragma unroll 16
      for (int i = lane; i < cnt; i += 32) s += __bfloat162float(buf[k & 1][i]);
    }
  }
  if (threadIdx.x < 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[blockIdx.x] = s;
  }
}

// loss = sum (y - t)^2 * scale, dY = 2 scale (y - t) (bf16, row-major and
// transposed); columns >= n are zero in dY.  A CTA takes 64 x 64 values
// through shared memory, so that the rows of both outputs are written
// whole (element by element the transposed stores took 53 us for 16,384 x
// 64).
__global__ void __launch_bounds__(256)
    k_loss_grad(const float *Yh, int64_t ldy, const float *Tg, int64_t ldt, int64_t m, int64_t n,
                int64_t n_pad, float scale, __nv_bfloat16 *dY, int64_t ld, __nv_bfloat16 *dYT,
                int64_t ldtt, float *loss) {
  __shared__ __nv_bfloat16 tile[64][66];
  __shared__ float part[8];
  const int64_t r0 = (int64_t)blockIdx.x * 64, c0 = (int64_t)blockIdx.y * 64;
  const int x = threadIdx.x & 63, y = threadIdx.x >> 6;
  float acc = 0.0f;
#pragma unroll 4
  for (int j = y; j < 64; j += 4) {
    const int64_t r = r0 + j, c = c0 + x;
    float g = 0.0f;
    if (r < m && c < n) {
      const float d = Yh[r * ldy + c] - Tg[r * ldt + c];
      acc += d * d;
      g = 2.0f * scale * d;
    }
    const __nv_bfloat16 gb = __float2bfloat16_rn(g);
    tile[j][x] = gb;
    if (r < m && c < n_pad) dY[r * ld + c] = gb;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
#pragma unroll 4
  for (int j = y; j < 64; j += 4)
    if (r0 + x < m && c0 + j < n_pad) dYT[(c0 + j) * ldtt + r0 + x] = tile[x][j];
  if (threadIdx.x == 0 && loss) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w];
    atomicAdd(loss, t * scale);
  }
}

// One tensor of an Adam step.
struct AdamTensor {
  float *p;
  const float *g;
  float *m, *v;
  __nv_bfloat16 *W, *WT;
  int64_t rows, cols, ldw, ldwt;
};
constexpr int ADAM_MAX = 16;
struct AdamSet {
  AdamTensor t[ADAM_MAX];
  int first[ADAM_MAX + 1];  // first CTA of each tensor
};

// All tensors of a step in one launch: a CTA belongs to one tensor.
__global__ void __launch_bounds__(256)
    k_adam(const __grid_constant__ AdamSet set, int count, float lr, float b1, float b2,
           float eps, float c1, float c2) {
  int q = 0;
  while (q + 1 < count && (int)blockIdx.x >= set.first[q + 1]) ++q;
  const AdamTensor &a = set.t[q];
  const int64_t n = a.rows * a.cols;
  const int64_t step = (int64_t)(set.first[q + 1] - set.first[q]) * blockDim.x;
  for (int64_t idx = (int64_t)(blockIdx.x - set.first[q]) * blockDim.x + threadIdx.x; idx < n;
       idx += step) {
    const float gi = a.g[idx];
    const float m = b1 * a.m[idx] + (1.0f - b1) * gi;
    const float v = b2 * a.v[idx] + (1.0f - b2) * gi * gi;
    a.m[idx] = m;
    a.v[idx] = v;
    const float w = a.p[idx] - lr * (m * c1) / (sqrtf(v * c2) + eps);
    a.p[idx] = w;
    const int64_t r = idx / a.cols, c = idx % a.cols;
    if (a.W) a.W[r * a.ldw + c] = __float2bfloat16_rn(w);
    if (a.WT) a.WT[c * a.ldwt + r] = __float2bfloat16_rn(w);
  }
}

// Features of state i: [(T - mu0)/sd0, (ln P - mu1)/sd1,
// (ln(Y_k + 1e-12) - mu_k)/sd_k for the N species], zero padding to ldx.
// out_of_box[i] = 1 when a feature leaves the training box [lo, hi].
__global__ void k_features(int64_t n, const double *T, const double *P, const double *Y,
                           int64_t ld, int nsp, const float *mu, const float *sd,
                           const float *lo, const float *hi, __nv_bfloat16 *X, int64_t ldx,
                           __nv_bfloat16 *XT, int64_t ldxt, int nfeat_pad,
                           unsigned char *out_of_box, float *raw) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    bool out = false;
    double ysum = 0.0;
    // eight features at a time: one 16-byte store of the row
    for (int f0 = 0; f0 < nfeat_pad; f0 += 8) {
      float x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int f = f0 + j;
        float v = 0.0f;
        if (f == 0) {
          v = (float)T[i];
        } else if (f == 1) {
          v = logf((float)P[i]);
        } else if (f < 2 + nsp) {
          const int k = f - 2;
          double y;
          if (k < nsp - 1) {
            y = Y[(int64_t)k * ld + i];
            ysum += y;
          } else {
            y = 1.0 - ysum;
          }
          v = logf(fmaxf((float)y, 0.0f) + 1.0e-12f);
        }
        if (f < 2 + nsp) {
          if (raw) raw[i * (2 + nsp) + f] = v;
          if (lo && (v < lo[f] || v > hi[f])) out = true;
          v = (v - mu[f]) / sd[f];
        }
        x[j] = v;
        if (XT) XT[(int64_t)f * ldxt + i] = __float2bfloat16_rn(v);
      }
      *reinterpret_cast<uint4 *>(X + i * ldx + f0) =
          make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]),
                     pack_bf16(x[6], x[7]));
    }
    if (out_of_box) out_of_box[i] = out;
  }
}

// v * 2^e as a double, by integer operations on v's fields (exact); values
// below the fp32 normal range give zero.
__device__ __forceinline__ double scale_to_double(float v, int e) {
  const uint32_t b = __float_as_uint(v);
  const int ef = (int)((b >> 23) & 0xFF);
  if (ef == 0) return 0.0;
  if (ef == 0xFF) return (double)v;
  const int ed = ef - 127 + 1023 + e;
  const uint64_t sign = (uint64_t)(b >> 31) << 63;
  if (ed >= 0x7FF) return __longlong_as_double((long long)(sign | 0x7FF0000000000000ull));
  if (ed <= 0) return __longlong_as_double((long long)sign);
  return __longlong_as_double(
      (long long)(sign | ((uint64_t)ed << 52) | ((uint64_t)(b & 0x7FFFFF) << 29)));
}

constexpr int MAX_ELEM = 8;

// Network output -> wdot.  With u_k = sign(y_k) expm1(|y_k|) (the rate in
// units of its scale s_k = sm_k 2^se_k), w_k = (u_k sm_k) 2^se_k in FP64.
// The state goes to the exact kernel when it is outside the training box or
// when its element residual
//   max_e |sum_k a_ek w_k| / sum_k a_ek (|w_k| + s_k)
// exceeds tol: conservation violated by more than tol of the rates' own
// size, or of their typical size where the rates are small.  The residual
// is formed in fp32 from cons[e][k] = a_ek s_k / max_j a_ej s_j, which
// keeps every term in range (rates reach 1e50 and beyond).
__global__ void k_output(int64_t n, const float *Yh, int64_t ldy, int nsp, const float *sm,
                         const int *se, const float *cons, int nelem, float tol,
                         const unsigned char *out_of_box, double *wdot, int64_t ld,
                         unsigned char *fallback) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float sum[MAX_ELEM], mag[MAX_ELEM];
#pragma unroll
    for (int e = 0; e < MAX_ELEM; ++e) sum[e] = mag[e] = 0.0f;
    for (int k = 0; k < nsp; ++k) {
      const float y = Yh[i * ldy + k];
      const float u = copysignf(expm1f(fabsf(y)), y);
      wdot[(int64_t)k * ld + i] = scale_to_double(u * sm[k], se[k]);
#pragma unroll
      for (int e = 0; e < MAX_ELEM; ++e) {
        if (e < nelem) {
          const float c = cons[e * nsp + k];
          sum[e] = fmaf(c, u, sum[e]);
          mag[e] = fmaf(c, fabsf(u) + 1.0f, mag[e]);
        }
      }
    }
    float worst = 0.0f;
#pragma unroll
    for (int e = 0; e < MAX_ELEM; ++e)
      if (e < nelem && mag[e] > 0.0f) worst = fmaxf(worst, fabsf(sum[e]) / mag[e]);
    const bool fb = !(worst <= tol) || (out_of_box && out_of_box[i]);
    fallback[i] = fb;
  }
}

// Rows i0 .. i0 + rows - 1 of the two members' outputs, read whole by the
// warp (lane = column): returns max_k |y_k,a - y_k,b| of row i0 + lane and,
// with mean, leaves the members' mean at mean[k * 33 + row].  NaN
// differences count as zero, as fmaxf drops them.
__device__ __forceinline__ float rows_of(const float *Ya, const float *Yb, int64_t ldy,
                                         int64_t i0, int rows, int nsp, int lane, float *mean) {
  float mine = 0.0f;
  for (int j0 = 0; j0 < rows; j0 += 4) {
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int k = lane; k < nsp; k += 32) {
      float a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // past the last row: that row again
        const int64_t i = i0 + (j0 + u < rows ? j0 + u : rows - 1);
        a[u] = __ldcs(Ya + i * ldy + k);
        b[u] = __ldcs(Yb + i * ldy + k);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        d[u] = fmaxf(d[u], fabsf(a[u] - b[u]));
        if (mean && j0 + u < rows) mean[k * 33 + j0 + u] = 0.5f * (a[u] + b[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // non-negative floats compare as their bits
      const float r = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(d[u])));
      if (lane == j0 + u) mine = r;
    }
  }
  return mine;
}

// Two-member output with an error gate.  The served y_k is the mean of the
// members' outputs; in y = sign(u) log1p|u| space a change dy moves w by
// |dy| (|w| + s) to first order, so an error in y is the reported error
// e = max_k |w_k - w_k,exact| / (|w_k,exact| + s_k).  The gate score of a
// state is
//   g = dweight log10(D + 1e-4) + E,   D = max_k |y_k,a - y_k,b|,
// the members' disagreement plus E = est[i * lde], the output of a network
// trained to predict log10(e + 1e-4) (omitted when est is NULL); the
// disagreement term is weighted by dweight (0 when the error network takes
// D as an input, see k_disagreement).  A state
// goes back to the exact kernel as in k_output, or when g > stol (NaN
// included).  gate[i] (optional) receives g, for calibrating stol.
// Bound by memory.  ROWS: a warp reads its 32 states' rows whole (lane =
// column; 32 lanes reading 32 rows fetch each sector up to eight times) and
// keeps the means in shared memory, column by state, for the sums over k that
// follow with lane = state in the order of k, four k's table entries and
// exponentials ahead of the sums; else a thread reads its state's row.  2^20
// states of 53 species: 342 us without, 308 with.
template <bool ROWS>
__global__ void __launch_bounds__(256)
    k_output2(int64_t n, const float *Ya, const float *Yb, int64_t ldy, int nsp,
              const float *sm, const int *se, const float *cons, int nelem, float tol,
              float dweight, const float *est, int64_t lde, float stol,
              const unsigned char *out_of_box, double *wdot, int64_t ld,
              unsigned char *fallback, float *gate) {
  extern __shared__ float mean[];
  const int lane = threadIdx.x & 31;
  float *col = mean + (ROWS ? (size_t)(threadIdx.x >> 5) * nsp * 33 : 0);
  const int64_t nwarp = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; i0 < n;
       i0 += nwarp * 32) {
    float d = 0.0f;
    if (ROWS) {
      const int rows = n - i0 < 32 ? (int)(n - i0) : 32;
      d = rows_of(Ya, Yb, ldy, i0, rows, nsp, lane, col);
      __syncwarp();
    }
    const int64_t i = i0 + lane;
    if (i < n) {
      float sum[MAX_ELEM], mag[MAX_ELEM];
#pragma unroll
      for (int e = 0; e < MAX_ELEM; ++e) sum[e] = mag[e] = 0.0f;
#pragma unroll 4
      for (int k = 0; k < nsp; ++k) {
        float y;
        if (ROWS) {
          y = col[k * 33 + lane];
        } else {
          const float ya = Ya[i * ldy + k], yb = Yb[i * ldy + k];
          d = fmaxf(d, fabsf(ya - yb));
          y = 0.5f * (ya + yb);
        }
        const float u = copysignf(expm1f(fabsf(y)), y);
        wdot[(int64_t)k * ld + i] = scale_to_double(u * sm[k], se[k]);
#pragma unroll
        for (int e = 0; e < MAX_ELEM; ++e) {
          if (e < nelem) {
            const float c = cons[e * nsp + k];
            sum[e] = fmaf(c, u, sum[e]);
            mag[e] = fmaf(c, fabsf(u) + 1.0f, mag[e]);
          }
        }
      }
      float worst = 0.0f;
#pragma unroll
      for (int e = 0; e < MAX_ELEM; ++e)
        if (e < nelem && mag[e] > 0.0f) worst = fmaxf(worst, fabsf(sum[e]) / mag[e]);
      const float g = dweight * log10f(d + 1.0e-4f) + (est ? est[i * lde] : 0.0f);
      const bool fb = !(worst <= tol) || !(g <= stol) || (out_of_box && out_of_box[i]);
      fallback[i] = fb;
      if (gate) gate[i] = g;
    }
    __syncwarp();
  }
}

// The members' disagreement D = max_k |y_k,a - y_k,b| as an input of the
// error network: X[i][col] = bf16((log10(D + 1e-4) - mu) / sd).
// ROWS: a warp takes `per` states' rows whole (see rows_of), else (per = 32) a
// thread a row.
template <bool ROWS>
__global__ void __launch_bounds__(256)
    k_disagreement(int64_t n, const float *Ya, const float *Yb, int64_t ldy, int nsp, float mu,
                   float sd, __nv_bfloat16 *X, int64_t ldx, int col, int per) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarp = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; i0 < n;
       i0 += nwarp * per) {
    const int rows = n - i0 < per ? (int)(n - i0) : per;
    float d = 0.0f;
    if (ROWS)
      d = rows_of(Ya, Yb, ldy, i0, rows, nsp, lane, nullptr);
    else if (lane < rows)
      for (int k = 0; k < nsp; ++k)
        d = fmaxf(d, fabsf(Ya[(i0 + lane) * ldy + k] - Yb[(i0 + lane) * ldy + k]));
    if (lane < rows)
      X[(i0 + lane) * ldx + col] = __float2bfloat16_rn((log10f(d + 1.0e-4f) - mu) / sd);
  }
}

// Indices of flagged states (order unspecified; one warp-aggregated atomic
// per warp).  count must be zero on entry.
__global__ void k_compact(int64_t n, const unsigned char *flag, int64_t *idx,
                          unsigned long long *count) {
  const int lane = threadIdx.x & 31;
  for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x; c0 < n;
       c0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = c0 + threadIdx.x;
    const bool f = i < n && flag[i];
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (!bal) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(count, (unsigned long long)__popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (f) idx[base + __popc(bal & ((1u << lane) - 1u))] = i;
  }
}

__global__ void k_gather(int64_t m, const int64_t *idx, const double *T, const double *P,
                         const double *Y, int64_t ld, int rows, double *Tc, double *Pc,
                         double *Yc, int64_t ldc) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < m;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx[j];
    Tc[j] = T[i];
    Pc[j] = P[i];
    for (int k = 0; k < rows; ++k) Yc[(int64_t)k * ldc + j] = Y[(int64_t)k * ld + i];
  }
}

__global__ void k_scatter(int64_t m, const int64_t *idx, const double *Wc, int64_t ldc,
                          int rows, double *W, int64_t ld) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < m;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx[j];
    for (int k = 0; k < rows; ++k) W[(int64_t)k * ld + i] = Wc[(int64_t)k * ldc + j];
  }
}

inline int grid1(int64_t n, int per = 256) {
  int64_t g = (n + per - 1) / per;
  if (g > 65535) g = 65535;
  return (int)(g < 1 ? 1 : g);
}

template <class Epi>
cudaError_t gemm_bn(const CUtensorMap &ta, const CUtensorMap &tb, int64_t M_pad, int64_t N_pad,
                    int64_t K, int bn, const Epi &epi, cudaStream_t s, int splits = 1) {
  // two-stage ring, 8 warps: two CTAs per SM (the network's K is small)
  switch (bn) {
    case 64: return launch_gemm<64, Epi, 2, 256>(ta, tb, M_pad, N_pad, K, epi, nullptr, s, splits);
    case 128: return launch_gemm<128, Epi, 2, 256>(ta, tb, M_pad, N_pad, K, epi, nullptr, s, splits);
    case 256: return launch_gemm<256, Epi, 2, 256>(ta, tb, M_pad, N_pad, K, epi, nullptr, s, splits);
    default: return cudaErrorInvalidValue;
  }
}

// Columns per CTA: the narrowest tile whose CTAs (m_tiles rows of 128 each)
// still run as one wave, two per SM, so that one's epilogue overlaps
// another's loads; re-reading A from L2 for more column tiles costs less
// than an idle SM, a second wave does not.
inline int pick_bn(int64_t n_pad, int64_t m_tiles) {
  int bn = n_pad % 256 == 0 ? 256 : n_pad % 128 == 0 ? 128 : n_pad % 64 == 0 ? 64 : 0;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return bn;
  while (bn > 64 && m_tiles * (n_pad / bn) * 2 <= 2 * (int64_t)sms) bn /= 2;
  return bn;
}

inline int bad(const char *fn) {
  char buf[160];
  snprintf(buf, sizeof buf, "%s: invalid argument (null pointer, size or alignment)", fn);
  return report(CRS_ERR_ARG, buf);
}

inline int done(cudaError_t e, const char *fn) {
  if (e == cudaSuccess) return CRS_OK;
  char buf[200];
  snprintf(buf, sizeof buf, "%s: %s", fn, cudaGetErrorString(e));
  return report(CRS_ERR_CUDA, buf);
}

}  // namespace mlp
}  // namespace crs

using namespace crs;
using mlp::bad;
using mlp::done;

extern "C" {

int crs_mlp_forward(const void *X, const void *W, const float *b, int64_t M_pad, int64_t N_pad,
                    int64_t K, int64_t M, int64_t N, int act, float *Z, int64_t ldz, void *A,
                    int64_t lda, void *AT, int64_t ldat, float *Y32, int64_t ldy,
                    void *stream) {
  const int bn = mlp::pick_bn(N_pad, M_pad / 128);
  if (!X || !W || M_pad % 128 || K % 64 || !bn || M > M_pad || N > N_pad) return bad(__func__);
  CUtensorMap ta, tb;
  if (!make_tmap_bf16(&ta, X, M_pad, K, 128) || !make_tmap_bf16(&tb, W, N_pad, K, bn))
    return bad(__func__);
  mlp::EpiForward epi{b, act, (int)M, (int)N, Z, ldz, static_cast<__nv_bfloat16 *>(A), lda,
                      static_cast<__nv_bfloat16 *>(AT), ldat, Y32, ldy};
  cudaError_t e = mlp::gemm_bn(ta, tb, M_pad, N_pad, K, bn, epi, static_cast<cudaStream_t>(stream));
  return done(e, __func__);
}

int crs_mlp_backward_data(const void *dZ, const void *WT, int64_t M_pad, int64_t Nin_pad,
                          int64_t Kout, int64_t M, int64_t Nin, const float *Zprev,
                          int64_t ldz, void *dZprev, int64_t ld, void *dZprevT, int64_t ldt,
                          void *stream) {
  const int bn = mlp::pick_bn(Nin_pad, M_pad / 128);
  if (!dZ || !WT || !Zprev || !dZprev || M_pad % 128 || Kout % 64 || !bn) return bad(__func__);
  CUtensorMap ta, tb;
  if (!make_tmap_bf16(&ta, dZ, M_pad, Kout, 128) || !make_tmap_bf16(&tb, WT, Nin_pad, Kout, bn))
    return bad(__func__);
  mlp::EpiBackwardData epi{Zprev, ldz, (int)M, (int)Nin, static_cast<__nv_bfloat16 *>(dZprev),
                           ld, static_cast<__nv_bfloat16 *>(dZprevT), ldt};
  cudaError_t e = mlp::gemm_bn(ta, tb, M_pad, Nin_pad, Kout, bn, epi, static_cast<cudaStream_t>(stream));
  return done(e, __func__);
}

int crs_mlp_backward_weight(const void *dZT, const void *AT, int64_t Nout_pad, int64_t Nin_pad,
                            int64_t M_pad, int64_t Nout, int64_t Nin, int splits,
                            float *partial, float *dW, void *stream) {
  const int bn = mlp::pick_bn(Nin_pad, Nout_pad / 128 * (splits > 0 ? splits : 1));
  if (!dZT || !AT || !partial || !dW || Nout_pad % 128 || M_pad % 64 || !bn || splits < 1 ||
      (M_pad / 64) % splits)
    return bad(__func__);
  CUtensorMap ta, tb;
  if (!make_tmap_bf16(&ta, dZT, Nout_pad, M_pad, 128) || !make_tmap_bf16(&tb, AT, Nin_pad, M_pad, bn))
    return bad(__func__);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  mlp::EpiPartial epi{partial, Nout_pad, Nin_pad};
  cudaError_t e = mlp::gemm_bn(ta, tb, Nout_pad, Nin_pad, M_pad, bn, epi, s, splits);
  if (e != cudaSuccess) return done(e, __func__);
  mlp::k_reduce_partials<<<mlp::grid1(Nout * Nin), 256, 0, s>>>(partial, splits, Nout_pad,
                                                                 Nin_pad, Nout, Nin, dW);
  return done(cudaGetLastError(), __func__);
}

int crs_mlp_row_sums(const void *X, int64_t ld, int64_t rows, int64_t m, float *out,
                     void *stream) {
  if (!X || !out || rows < 0 || m < 0 || ld < m) return bad(__func__);
  if (rows == 0) return CRS_OK;
  // (256 rows of 4,096: 6.2 us with a warp per row, 4.2 with a CTA; of 1,024: 3.3
  // to 4.1 and 3.9; 4,096 rows of 128: 3.5 and 8.2, of 4,096: 8.3 and 12.3)
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (m > 2048 && rows <= 1024)
    mlp::k_row_sums<<<(unsigned)rows, 256, 0, s>>>(static_cast<const __nv_bfloat16 *>(X), ld, m,
                                                   out);
  else
    mlp::k_row_sums_short<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>(
        static_cast<const __nv_bfloat16 *>(X), ld, rows, m, out);
  return done(cudaGetLastError(), __func__);
}

int crs_mlp_loss_grad(const float *Yh, int64_t ldy, const float *Tg, int64_t ldt, int64_t m,
                      int64_t n, int64_t n_pad, float scale, void *dY, int64_t ld, void *dYT,
                      int64_t ldtt, float *loss, void *stream) {
  if (!Yh || !Tg || !dY || !dYT || m < 0 || n > n_pad) return bad(__func__);
  if (m == 0 || n_pad == 0) return CRS_OK;
  const dim3 grid((unsigned)((m + 63) / 64), (unsigned)((n_pad + 63) / 64));
  mlp::k_loss_grad<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      Yh, ldy, Tg, ldt, m, n, n_pad, scale, static_cast<__nv_bfloat16 *>(dY), ld,
      static_cast<__nv_bfloat16 *>(dYT), ldtt, loss);
  return done(cudaGetLastError(), __func__);
}

int crs_adam_steps(int count, float *const *p, const float *const *g, float *const *m,
                   float *const *v, const int64_t *rows, const int64_t *cols, float lr, float b1,
                   float b2, float eps, int step, void *const *W, const int64_t *ldw,
                   void *const *WT, const int64_t *ldwt, void *stream) {
  if (count < 0 || count > mlp::ADAM_MAX || !p || !g || !m || !v || !rows || !cols || !W ||
      !ldw || !WT || !ldwt || step < 1)
    return bad(__func__);
  mlp::AdamSet set{};
  int ctas = 0;
  for (int q = 0; q < count; ++q) {
    if (!p[q] || !g[q] || !m[q] || !v[q] || rows[q] < 0 || cols[q] < 0) return bad(__func__);
    set.t[q] = mlp::AdamTensor{p[q], g[q], m[q], v[q], static_cast<__nv_bfloat16 *>(W[q]),
                               static_cast<__nv_bfloat16 *>(WT[q]), rows[q], cols[q], ldw[q],
                               ldwt[q]};
    set.first[q] = ctas;
    ctas += mlp::grid1(rows[q] * cols[q]);
  }
  for (int q = count; q <= mlp::ADAM_MAX; ++q) set.first[q] = ctas;
  if (ctas == 0) return CRS_OK;
  const float c1 = 1.0f / (1.0f - powf(b1, (float)step));
  const float c2 = 1.0f / (1.0f - powf(b2, (float)step));
  mlp::k_adam<<<(unsigned)ctas, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      set, count, lr, b1, b2, eps, c1, c2);
  return done(cudaGetLastError(), __func__);
}

int crs_adam_step(float *p, const float *g, float *m, float *v, int64_t rows, int64_t cols,
                  float lr, float b1, float b2, float eps, int step, void *W, int64_t ldw,
                  void *WT, int64_t ldwt, void *stream) {
  if (!p || !g || !m || !v || rows < 0 || cols < 0 || step < 1) return bad(__func__);
  return crs_adam_steps(1, &p, &g, &m, &v, &rows, &cols, lr, b1, b2, eps, step, &W, &ldw, &WT,
                        &ldwt, stream);
}

int crs_surrogate_features(int64_t n, const double *T, const double *P, const double *Y,
                           int64_t ld, int nsp, const float *mu, const float *sd,
                           const float *lo, const float *hi, void *X, int64_t ldx, void *XT,
                           int64_t ldxt, int nfeat_pad, unsigned char *out_of_box, float *raw,
                           void *stream) {
  if (n < 0 || !T || !P || !Y || !mu || !sd || !X || nfeat_pad < 2 + nsp || nfeat_pad % 8 ||
      ldx % 8 || ldx < nfeat_pad || (reinterpret_cast<uintptr_t>(X) & 15) || ld < n)
    return bad(__func__);
  if (n == 0) return CRS_OK;
  mlp::k_features<<<mlp::grid1(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      n, T, P, Y, ld, nsp, mu, sd, lo, hi, static_cast<__nv_bfloat16 *>(X), ldx,
      static_cast<__nv_bfloat16 *>(XT), ldxt, nfeat_pad, out_of_box, raw);
  return done(cudaGetLastError(), __func__);
}

int crs_surrogate_output(int64_t n, const float *Yh, int64_t ldy, int nsp, const float *scale_m,
                         const int *scale_e, const float *cons, int nelem, float tol,
                         const unsigned char *out_of_box, double *wdot, int64_t ld,
                         unsigned char *fallback, void *stream) {
  if (n < 0 || !Yh || !scale_m || !scale_e || !wdot || !fallback || (nelem && !cons) ||
      nelem < 0 || nelem > mlp::MAX_ELEM || ld < n || ldy < nsp)
    return bad(__func__);
  if (n == 0) return CRS_OK;
  mlp::k_output<<<mlp::grid1(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      n, Yh, ldy, nsp, scale_m, scale_e, cons, nelem, tol, out_of_box, wdot, ld, fallback);
  return done(cudaGetLastError(), __func__);
}

int crs_surrogate_output2(int64_t n, const float *Ya, const float *Yb, int64_t ldy, int nsp,
                          const float *scale_m, const int *scale_e, const float *cons, int nelem,
                          float tol, float dweight, const float *est, int64_t lde, float stol,
                          const unsigned char *out_of_box, double *wdot, int64_t ld,
                          unsigned char *fallback, float *gate, void *stream) {
  if (n < 0 || !Ya || !Yb || !scale_m || !scale_e || !wdot || !fallback ||
      (nelem && !cons) || nelem < 0 || nelem > mlp::MAX_ELEM || ld < n || ldy < nsp ||
      (est && lde < 1))
    return bad(__func__);
  if (n == 0) return CRS_OK;
  // Rows read whole pay from 32 species on (below, lanes idle: 10 species,
  // 2^20 states 58 us with a row per thread, 101 so; 32: 304 and 176), in small
  // batches from 48 (40 species, 500 states: 18.5 and 20.1), as long as the
  // columns of means leave room for two CTAs of eight warps per SM (96 species,
  // 2^20 states: 897 and 642; 112: 825 and 1,363), or all the states are on chip
  // with one (300 species, 8,192 states: 137 and 114; 65,536: 198 and 340).
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return done(e, __func__);
  const size_t per_warp = (size_t)(nsp > 0 ? nsp : 1) * 33 * sizeof(float);
  const size_t fit = ((size_t)200 << 10) / per_warp;
  const int nw = fit < 8 ? (int)fit : 8;
  const bool rows = (nsp >= 48 || (nsp >= 32 && n >= 32768)) &&
                    (fit >= 16 || n <= (int64_t)sms * nw * 32);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows) {
    e = raise_smem_limit(mlp::k_output2<true>);
    if (e != cudaSuccess) return done(e, __func__);
    mlp::k_output2<true><<<mlp::grid1(n, nw * 32), nw * 32, nw * per_warp, s>>>(
        n, Ya, Yb, ldy, nsp, scale_m, scale_e, cons, nelem, tol, dweight, est, lde, stol,
        out_of_box, wdot, ld, fallback, gate);
  } else {
    mlp::k_output2<false><<<mlp::grid1(n), 256, 0, s>>>(
        n, Ya, Yb, ldy, nsp, scale_m, scale_e, cons, nelem, tol, dweight, est, lde, stol,
        out_of_box, wdot, ld, fallback, gate);
  }
  return done(cudaGetLastError(), __func__);
}

int crs_surrogate_disagreement(int64_t n, const float *Ya, const float *Yb, int64_t ldy,
                               int nsp, float mu, float sd, void *X, int64_t ldx, int col,
                               void *stream) {
  if (n < 0 || !Ya || !Yb || !X || ldy < nsp || col < 0 || col >= ldx || !(sd > 0.0f))
    return bad(__func__);
  if (n == 0) return CRS_OK;
  // rows read whole from 32 species on (2^20 states: 10 species 30 us with a row
  // per thread, 68 so; 32: 232 and 72); eight rows per warp where that does not
  // fill the chip
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (nsp >= 32) {
    const int per = n < 32768 ? 8 : 32;
    mlp::k_disagreement<true><<<mlp::grid1(n, 4 * per), 128, 0, s>>>(
        n, Ya, Yb, ldy, nsp, mu, sd, static_cast<__nv_bfloat16 *>(X), ldx, col, per);
  } else {
    mlp::k_disagreement<false><<<mlp::grid1(n), 256, 0, s>>>(
        n, Ya, Yb, ldy, nsp, mu, sd, static_cast<__nv_bfloat16 *>(X), ldx, col, 32);
  }
  return done(cudaGetLastError(), __func__);
}

int crs_select(int64_t n, const unsigned char *flag, int64_t *idx, int64_t *count, void *stream) {
  if (n < 0 || !flag || !idx || !count) return bad(__func__);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int64_t), s);
  if (e != cudaSuccess || n == 0) return done(e, __func__);
  mlp::k_compact<<<mlp::grid1(n), 256, 0, s>>>(n, flag, idx,
                                               reinterpret_cast<unsigned long long *>(count));
  return done(cudaGetLastError(), __func__);
}

int crs_gather_states(int64_t m, const int64_t *idx, const double *T, const double *P,
                      const double *Y, int64_t ld, int rows, double *Tc, double *Pc, double *Yc,
                      int64_t ldc, void *stream) {
  if (m < 0 || !idx || ldc < m) return bad(__func__);
  if (m == 0) return CRS_OK;
  mlp::k_gather<<<mlp::grid1(m), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      m, idx, T, P, Y, ld, rows, Tc, Pc, Yc, ldc);
  return done(cudaGetLastError(), __func__);
}

int crs_scatter_wdot(int64_t m, const int64_t *idx, const double *Wc, int64_t ldc, int rows,
                     double *W, int64_t ld, void *stream) {
  if (m < 0 || !idx || ldc < m) return bad(__func__);
  if (m == 0) return CRS_OK;
  mlp::k_scatter<<<mlp::grid1(m), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      m, idx, Wc, ldc, rows, W, ld);
  return done(cudaGetLastError(), __func__);
}

}  // extern "C"
