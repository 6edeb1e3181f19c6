// Slice-pipeline steps around gridrec, on the device (decarlof/projects):
//   ring suppression        RingCorrectionSinogram  gridrec/GPU/tomo_recon.cpp:3905-3968
//   sub-pixel shift + pad   GridRecSlices           gridrec/GPU/tomo_recon.cpp:3708-3810
//                           (same code in find_shift/src/main/find_shift.cpp:1729-1808)
//   centre crop             GridRecSlices           gridrec/GPU/tomo_recon.cpp:3855-3862
//   circular crop           output stage            gridrec/GPU/tomo_recon.cpp:2150-2165
//   histogram entropy       entropy()               find_shift/src/main/find_shift.cpp:2078-2115
//   centre search           entropy refinement      find_shift/src/main/find_shift.cpp:1653-1900
// Sinograms are n_ang rows of n_det floats, slices contiguous.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "gr_internal.h"

namespace gr {
namespace {

constexpr int kPrepThreads = 256;
constexpr int kMaxBins = 50000;

__device__ __forceinline__ float block_sum(float v, float* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float s = 0.f;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (int)(blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;  // valid in thread 0
}

__device__ __forceinline__ double block_sum_d(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (int)(blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}

// ---------------------------------------------------------------------------
// Ring suppression.  Each of `iterations` rounds, per slice:
//   r_i = mean_j x_ij,  g = mean_i r_i,  v_ij = x_ij g / r_i   (rows with r_i = 0 kept)
//   c_j = mean_i v_ij,  t_j = c_j - (c_{j-1} + c_j + c_{j+1}) / 3   (t_0 = t_{n-1} = 0)
//   x_ij <- v_ij - coeff t_j  where positive, else 0
// Two launches per round: the row update fused with the next round's row means
// and column partial sums over chunks of rows, then the column means.  The
// first round's partials come from a pass over the input.  The
// renormalised value is formed as (x g) / r in float, the reference's expression.

// Rows per chunk of the column passes over rows wider than 4096 or not made of aligned
// 16-byte pieces (32: measured fastest of 4..32 at 16 x 2048 x 1500; more row chunks add
// partial-sum traffic, fewer leave SMs idle).
constexpr int kRingRows = 32;

int ring_chunks(int n_ang) { return (n_ang + kRingRows - 1) / kRingRows; }

__global__ void ring_rowmean_kernel(const float* data, float* rowmean, int n_det, int n_ang) {
  __shared__ float red[32];
  const int i = blockIdx.x, s = blockIdx.y;
  const float* row = data + ((size_t)s * n_ang + i) * n_det;
  float acc = 0.f;
  for (int j = threadIdx.x; j < n_det; j += blockDim.x) acc += row[j];
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) rowmean[(size_t)s * n_ang + i] = acc / n_det;
}

// g, the mean of a slice's row means.  Summed in FP64: an error of g scales the whole slice in
// every round (20 rounds' error against float64 at 1024 x 720 x 16: 3.5e-7 with FP32 sums of g,
// 2.2e-7).
__device__ __forceinline__ float slice_gmean(const float* rm, int n_ang) {
  __shared__ float g_s;
  __shared__ double red[32];
  double acc = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < n_ang; i += blockDim.x) acc += rm[i];
  acc = block_sum_d(acc, red);
  if (threadIdx.x == 0) g_s = (float)(acc / n_ang);
  __syncthreads();
  return g_s;
}

__global__ void ring_colpart_kernel(const float* data, const float* rowmean, float* part,
                                    float* gmean, int n_det, int n_ang, int rows_per_chunk) {
  const int r = blockIdx.y, s = blockIdx.z, R = gridDim.y;
  const float* rm = rowmean + (size_t)s * n_ang;
  const float g = slice_gmean(rm, n_ang);
  if (threadIdx.x == 0 && blockIdx.x == 0 && r == 0) gmean[s] = g;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_det) return;
  const int i0 = r * rows_per_chunk, i1 = min(n_ang, i0 + rows_per_chunk);
  const float* x = data + (size_t)s * n_ang * n_det + j;
  float acc = 0.f;
  for (int i = i0; i < i1; ++i) {
    const float ri = rm[i];
    const float v = x[(size_t)i * n_det];
    acc += ri != 0.f ? __fdiv_rn(__fmul_rn(v, g), ri) : v;
  }
  part[((size_t)s * R + r) * n_det + j] = acc;
}

// Column means c_j = g / n_ang * sum_q part[q][j] (32 columns x 16 chunk
// strides per block).  scaled = 1: partials already include g (first round,
// sums of v); scaled = 0: partials are sums of x / r_i and g, the mean of the
// row means, is formed here and recorded for the next update.
constexpr int kColStrides = 16;

__global__ void __launch_bounds__(32 * kColStrides) ring_colmean_kernel(const float* part, const float* rowmean,
                                                          float* colmean, float* gmean, int n_det,
                                                          int n_ang, int R, int scaled) {
  __shared__ float acc_s[kColStrides][33];
  const int s = blockIdx.y;
  float g = 1.f;
  if (!scaled) {
    g = slice_gmean(rowmean + (size_t)s * n_ang, n_ang);
    if (threadIdx.x == 0 && blockIdx.x == 0) gmean[s] = g;
  }
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + tx;
  float acc = 0.f;
  if (j < n_det) {
    const float* p = part + (size_t)s * R * n_det + j;
#pragma unroll 4
    for (int q = ty; q < R; q += kColStrides) acc += p[(size_t)q * n_det];
  }
  acc_s[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && j < n_det) {
    float c = 0.f;
    for (int q = 0; q < kColStrides; ++q) c += acc_s[q][tx];
    colmean[(size_t)s * n_det + j] = c * g / n_ang;
  }
}

// One round on rows [r * rows_per_chunk, ...) of slice s, all columns, fused
// with the next round's column partials:
//   t_j = c_j - (c_{j-1} + c_j + c_{j+1}) / 3 (0 at both edges),
//   x <- max((x g) / r_i - coeff t_j, 0),  r_i <- mean of the new row,
//   part[j] = sum over the chunk of x_new / r_i.
// After a round every value is >= 0, so a row with r_i = 0 is all zeros and
// adds nothing whether scaled or not.  KPT columns per thread, RB rows per
// barrier (warp partials double-buffered).
template <int KPT, int RB>
__global__ void __launch_bounds__(kPrepThreads) ring_round_kernel(
    float* data, float* rowmean, const float* colmean, const float* gmean, float* part, int n_det,
    int n_ang, int rows_per_chunk, float coeff) {
  constexpr int NW = kPrepThreads / 32;
  __shared__ float red[2][RB][NW];
  const int r = blockIdx.x, s = blockIdx.y, R = gridDim.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float g = gmean[s];
  const float* c = colmean + (size_t)s * n_det;
  float d[KPT], acc[KPT];
#pragma unroll
  for (int k = 0; k < KPT; ++k) {
    const int j = threadIdx.x + k * kPrepThreads;
    float t = 0.f;
    if (j > 0 && j < n_det - 1) t = c[j] - (c[j - 1] + c[j] + c[j + 1]) / 3.f;
    d[k] = __fmul_rn(t, coeff);
    acc[k] = 0.f;
  }
  float* rm = rowmean + (size_t)s * n_ang;
  const int i0 = r * rows_per_chunk, i1 = min(n_ang, i0 + rows_per_chunk);
  int buf = 0;
  for (int ib = i0; ib < i1; ib += RB, buf ^= 1) {
    float y[RB][KPT];
    float ri[RB], sum[RB];
    // all loads of the RB rows first, so they are in flight together
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = ib + b;
      ri[b] = i < i1 ? rm[i] : 0.f;
      const float* row = data + ((size_t)s * n_ang + i) * n_det;
#pragma unroll
      for (int k = 0; k < KPT; ++k) {
        const int j = threadIdx.x + k * kPrepThreads;
        y[b][k] = (i < i1 && j < n_det) ? row[j] : 0.f;
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = ib + b;
      sum[b] = 0.f;
      float* row = data + ((size_t)s * n_ang + i) * n_det;
#pragma unroll
      for (int k = 0; k < KPT; ++k) {
        const int j = threadIdx.x + k * kPrepThreads;
        if (i < i1 && j < n_det) {
          const float x = y[b][k];
          // A zero sample skips the division: for finite g its quotient is +-0,
          // and +-0 - d rounds to the same float for either sign, so the result
          // is the same.  Zeros are common after a round's clamp, and warps
          // holding some of them ran up to 25 % slower through the division
          // (measured on phantom sinograms).
          const float v = (ri[b] != 0.f && x != 0.f) ? __fdiv_rn(__fmul_rn(x, g), ri[b]) : x;
          y[b][k] = __fsub_rn(v, d[k]) > 0.f ? __fsub_rn(v, d[k]) : 0.f;
          row[j] = y[b][k];
        }
        sum[b] += y[b][k];
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float v = sum[b];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[buf][b][w] = v;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float tot = 0.f;
#pragma unroll
      for (int q = 0; q < NW; ++q) tot += red[buf][b][q];
      const float rn = tot / n_det;
      const int i = ib + b;
      if (i < i1) {
        if (threadIdx.x == 0) rm[i] = rn;
        if (rn != 0.f) {
          const float inv = 1.f / rn;
#pragma unroll
          for (int k = 0; k < KPT; ++k) acc[k] += y[b][k] * inv;
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KPT; ++k) {
    const int j = threadIdx.x + k * kPrepThreads;
    if (j < n_det) part[((size_t)s * R + r) * n_det + j] = acc[k];
  }
}

// a / b correctly rounded for every a that is 0 or in [kDivLo, 2^100] and b in
// [2^-40, 2^40], with y = RN(1 / b): RN(a y) is within 2 ulp of a / b, one residual step
// brings it within 1 ulp, and a second one rounds correctly (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990; the residuals are
// exact in this range).  One reciprocal serves a row.
constexpr float kDivLo = 0x1p-60f;
__device__ __forceinline__ float div_by(float a, float b, float y) {
  float q = __fmul_rn(a, y);
  q = __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
  return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

// Threads of a block for rows of n_det, and blocks per SM at the kernel's registers.
constexpr int ring_threads(int n_det) { return n_det <= 2048 ? 128 : 256; }
constexpr int ring_blocks(int threads) { return threads == 128 ? 5 : 2; }

// Column sums of the vector kernels: a thread adds kRingGroup rows in FP32, then adds that sum
// to an FP64 one that starts at kRingSum0, rounding down.  While a column's sum of x / r stays
// below 2^21 in magnitude, every such addition keeps the multiples of 2^-30 below the sum
// (kRingSum0 + sum lies in [2^22, 2^23), one binade), so the additions are exact in any order:
// how a slice's rows are divided among blocks, which follows from the slices of the call, does
// not show in its bits.  (Sums beyond that are FP64 sums of the usual kind.)
constexpr int kRingGroup = 4;
constexpr double kRingSum0 = 6291456.0;  // 1.5 * 2^22

// The same round on rows of whole aligned 16-byte pieces: thread t of NT owns the pieces
// t, t + NT, ... of a row (KV of them), so a row of 2048 costs four loads and four stores
// per thread, the work per row (means, reciprocals, exchanges) is shared by 16 samples
// of a thread, and rows whose mean and data are in div_by's range divide by one
// reciprocal.  kFirst: the data may be negative (the first round), where the row mean
// does not bound the samples and every division is the general one.  kStart: no update,
// only the input's row means and column partials, with a flag per block for a row of mean
// 0 that is not all zero (its samples enter the column means unscaled:
// ring_first_colmean_kernel does such slices).
// Bound: DRAM once a call's slices exceed L2, then issue (17 instructions per sample, and
// 50 per thread and row group for the FP64 sums).  16 slices of 2048 x 1500: 67.7 us per
// round for 393 MB read and written, and 7.0 for the means; 20 rounds 2.42 -> 1.48 ms against
// the scalar kernels, one slice 0.89 -> 0.35 ms.  (Column sums kept in FP32 over a block's rows
// take 64.3 us per round, but their bits follow the number of slices of the call; FP32 sums over
// fixed chunks of 8, 12 or 16 rows 1.74, 1.60 and 1.71 ms for the 20 rounds; writing a block's
// only or last group without the shared copy 69.2 us.)  4 slices of 3000 x 1200, which fit L2:
// 0.71 ms, 0.64 with FP32 sums.  256 threads of half the pieces cost 74 us per round, groups of
// slices that fit L2 more than one wave of all slices (80 MB groups 2.30 ms for the call).
enum RingMode { kStart, kFirst, kLater };
template <int NT, int KV, int RB, RingMode kMode>
__global__ void __launch_bounds__(NT, ring_blocks(NT)) ring_round_vec_kernel(
    float* data, float* rowmean, const float* colmean, const float* gmean, const float* cscale,
    double* part, int n_det, int n_ang, int rows_per_block, float coeff, bool backward, int* flags) {
  constexpr int NW = NT / 32, GB = kRingGroup / RB;  // batches of RB rows in a group
  __shared__ __align__(16) float red[2][RB][NW];
  __shared__ double2 colsum[KV * 2][NT];  // a thread's own columns: pairs 2 k and 2 k + 1
  const int r = blockIdx.x, s = blockIdx.y, R = gridDim.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float g = kMode == kStart ? 0.f : gmean[s], cs = kMode == kStart ? 0.f : cscale[s];
  const float* c = colmean + (size_t)s * n_det;
  float d[KV][4], acc[KV][4];
  bool odd_row = false;
#pragma unroll
  for (int k = 0; k < KV; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = 4 * (threadIdx.x + k * NT) + e;
      float t = 0.f;
      if (kMode != kStart && j > 0 && j < n_det - 1) t = c[j] - (c[j - 1] + c[j] + c[j + 1]) / 3.f;
      d[k][e] = __fmul_rn(__fmul_rn(t, cs), coeff);
      acc[k][e] = 0.f;
    }
#pragma unroll
  for (int k = 0; k < 2 * KV; ++k) colsum[k][threadIdx.x] = make_double2(kRingSum0, kRingSum0);
  float* rm = rowmean + (size_t)s * n_ang;
  const int i0 = r * rows_per_block, i1 = min(n_ang, i0 + rows_per_block);
  const bool g_ok = !(kMode != kLater) && g >= 0x1p-40f && g <= 0x1p40f;
  // odd rounds walk the rows backwards: what the previous round wrote last is in L2
  const int nb = (i1 - i0 + RB - 1) / RB;
  int buf = 0;
  for (int t = 0; t < nb; ++t, buf ^= 1) {
    const int bt = backward ? nb - 1 - t : t, ib = i0 + bt * RB;
    float4 y[RB][KV];
    float ri[RB], sum[RB];
    // all loads of the RB rows first, so they are in flight together
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = ib + b;
      ri[b] = kMode != kStart && i < i1 ? rm[i] : 0.f;
      const float4* row = reinterpret_cast<const float4*>(data + ((size_t)s * n_ang + i) * n_det);
#pragma unroll
      for (int k = 0; k < KV; ++k) {
        const int q = threadIdx.x + k * NT;
        y[b][k] = (i < i1 && 4 * q < n_det) ? row[q] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = ib + b;
      sum[b] = 0.f;
      float4* row = reinterpret_cast<float4*>(data + ((size_t)s * n_ang + i) * n_det);
      // data >= 0: no sample exceeds n_det times its row's mean
      const bool fast = g_ok && ri[b] >= 0x1p-40f && ri[b] <= 0x1p40f;
      const float inv = __frcp_rn(fast ? ri[b] : 1.f);
#pragma unroll
      for (int k = 0; k < KV; ++k) {
        const int q = threadIdx.x + k * NT;
        float* x = reinterpret_cast<float*>(&y[b][k]);
        if (kMode == kStart) {
          sum[b] += (x[0] + x[1]) + (x[2] + x[3]);
          continue;
        }
        float v[4];
        bool ok = fast;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float a = __fmul_rn(x[e], g);
          v[e] = div_by(a, ri[b], inv);
          ok = ok && __float_as_uint(a) - 1u >= __float_as_uint(kDivLo) - 1u;  // 0 or >= kDivLo
        }
        if (!ok) {
#pragma unroll
          for (int e = 0; e < 4; ++e)  // zeros as in ring_round_kernel
            v[e] = (ri[b] != 0.f && x[e] != 0.f) ? __fdiv_rn(__fmul_rn(x[e], g), ri[b]) : x[e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[e] = fmaxf(__fsub_rn(v[e], d[k][e]), 0.f);  // NaN gives 0, as z > 0 ? z : 0
        }
        if (i < i1 && 4 * q < n_det) {
          row[q] = y[b][k];
          sum[b] += (x[0] + x[1]) + (x[2] + x[3]);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float v = sum[b];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[buf][b][w] = v;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float tot = 0.f;
#pragma unroll
      for (int q = 0; q < NW; q += 4) {
        const float4 p = *reinterpret_cast<const float4*>(&red[buf][b][q]);
        tot += (p.x + p.y) + (p.z + p.w);
      }
      const float rn = tot / n_det;
      const int i = ib + b;
      if (i < i1) {
        if (threadIdx.x == 0) rm[i] = rn;
        if (kMode == kStart && rn == 0.f) {
#pragma unroll
          for (int k = 0; k < KV; ++k)
            odd_row = odd_row || y[b][k].x != 0.f || y[b][k].y != 0.f || y[b][k].z != 0.f || y[b][k].w != 0.f;
        }
        if (rn != 0.f) {
          const float inv = 1.f / rn;
#pragma unroll
          for (int k = 0; k < KV; ++k) {
            acc[k][0] += y[b][k].x * inv;
            acc[k][1] += y[b][k].y * inv;
            acc[k][2] += y[b][k].z * inv;
            acc[k][3] += y[b][k].w * inv;
          }
        }
      }
    }
    if (backward ? bt % GB == 0 : (bt % GB == GB - 1 || t == nb - 1)) {  // a group's last rows
#pragma unroll
      for (int k = 0; k < 2 * KV; ++k) {
        float* g2 = &acc[k / 2][k % 2 * 2];
        double2 c2 = colsum[k][threadIdx.x];
        c2.x = __dadd_rd(c2.x, (double)g2[0]);
        c2.y = __dadd_rd(c2.y, (double)g2[1]);
        colsum[k][threadIdx.x] = c2;
        g2[0] = g2[1] = 0.f;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 2 * KV; ++k) {
    const int q = threadIdx.x + k / 2 * NT;
    const double2 c2 = colsum[k][threadIdx.x];
    if (4 * q < n_det)
      reinterpret_cast<double2*>(part + ((size_t)s * R + r) * n_det)[2 * q + k % 2] =
          make_double2(c2.x - kRingSum0, c2.y - kRingSum0);
  }
  if (kMode == kStart) {
    const bool any = __syncthreads_or(odd_row);
    if (threadIdx.x == 0) flags[(size_t)s * R + r] = any;
  }
}

// Whether some block of a slice met a row of mean 0 that is not all zero.  Called by the
// whole block.
__device__ __forceinline__ bool slice_flagged(const int* flags, int R) {
  bool f = false;
  for (int q = threadIdx.x; q < R; q += blockDim.x) f = f || flags[q] != 0;
  return __syncthreads_or(f);
}

// Means of the vector kernels.  A block takes COLS columns in STR strides: colmean_j = sum_q
// part[q][j] / n_ang (exact sums: any split gives the same bits), the factor g of the column
// mean being left to the reader (cscale).  The last block of a slice forms g, the mean of its
// row means, meanwhile.  flags given (after the start pass): no column means and a factor 1
// for flagged slices.
template <int COLS, int STR>
__global__ void __launch_bounds__(COLS * STR) ring_colmean_vec_kernel(
    const double* part, const float* rowmean, float* colmean, float* gmean, float* cscale, int n_det,
    int n_ang, int R, const int* flags) {
  __shared__ double acc_s[STR][COLS + 1];
  const int s = blockIdx.y;
  const bool flagged = flags && slice_flagged(flags + (size_t)s * R, R);
  if (blockIdx.x == gridDim.x - 1) {
    const float g = slice_gmean(rowmean + (size_t)s * n_ang, n_ang);
    if (threadIdx.x == 0) gmean[s] = g, cscale[s] = flagged ? 1.f : g;
    return;
  }
  if (flagged) return;
  const int tx = threadIdx.x % COLS, ty = threadIdx.x / COLS;
  const int j0 = blockIdx.x * COLS;
  double acc = 0.0;
  if (j0 + tx < n_det) {
    const double* p = part + (size_t)s * R * n_det + j0 + tx;
#pragma unroll 8
    for (int q = ty; q < R; q += STR) acc += p[(size_t)q * n_det];
  }
  acc_s[ty][tx] = acc;
  __syncthreads();
  const int j = j0 + threadIdx.x / STR;  // STR lanes per column
  double c = acc_s[threadIdx.x % STR][threadIdx.x / STR];
#pragma unroll
  for (int o = STR / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (threadIdx.x % STR == 0 && j < n_det) colmean[(size_t)s * n_det + j] = (float)(c / n_ang);
}

// First column means of flagged slices (those of the start pass leave out what a row of mean
// 0 adds): ring_colpart_kernel's and ring_colmean_kernel's sums in one pass.
__global__ void __launch_bounds__(32 * kColStrides) ring_first_colmean_kernel(
    const float* data, const float* rowmean, float* colmean, int n_det, int n_ang, int R,
    const int* flags) {
  __shared__ float acc_s[kColStrides][33];
  const int s = blockIdx.y;
  if (!slice_flagged(flags + (size_t)s * R, R)) return;
  const float* rm = rowmean + (size_t)s * n_ang;
  const float g = slice_gmean(rm, n_ang);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + tx;
  float acc = 0.f;
  if (j < n_det)
    for (int q = ty; q * kRingRows < n_ang; q += kColStrides) {
      float p = 0.f;
      for (int i = q * kRingRows; i < min(n_ang, (q + 1) * kRingRows); ++i) {
        const float x = data[((size_t)s * n_ang + i) * n_det + j];
        const float ri = rm[i];
        p += ri != 0.f ? __fdiv_rn(__fmul_rn(x, g), ri) : x;
      }
      acc += p;
    }
  acc_s[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && j < n_det) {
    float c = 0.f;
    for (int q = 0; q < kColStrides; ++q) c += acc_s[q][tx];
    colmean[(size_t)s * n_det + j] = c / n_ang;
  }
}

__global__ void ring_update_kernel(float* data, float* rowmean, const float* colmean,
                                   const float* gmean, int n_det, int n_ang, float coeff) {
  __shared__ float red[32];
  const int i = blockIdx.x, s = blockIdx.y;
  float* row = data + ((size_t)s * n_ang + i) * n_det;
  const float* c = colmean + (size_t)s * n_det;
  const float ri = rowmean[(size_t)s * n_ang + i];
  const float g = gmean[s];
  float acc = 0.f;
  for (int j = threadIdx.x; j < n_det; j += blockDim.x) {
    const float t = (j > 0 && j < n_det - 1) ? c[j] - (c[j - 1] + c[j] + c[j + 1]) / 3.f : 0.f;
    const float x = row[j];
    const float v = (ri != 0.f && x != 0.f) ? __fdiv_rn(__fmul_rn(x, g), ri) : x;  // as above
    const float d = __fmul_rn(t, coeff);
    const float y = __fsub_rn(v, d) > 0.f ? __fsub_rn(v, d) : 0.f;
    row[j] = y;
    acc += y;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) rowmean[(size_t)s * n_ang + i] = acc / n_det;
}

// ---------------------------------------------------------------------------
// Sub-pixel shift and half padding.  Slice s is shifted by x0 = xoff[s].  Column k of the
// input row maps to kp = k + pad (pad = n_det / 2) and takes
//   kk = k - x0,  n = floor(kk),  in[clamp(n)] (n + 1 - kk) + in[clamp(n + 1)] (kk - n)
// with indices clamped to [0, n_det); columns left of pad repeat column pad,
// the pad columns right of pad + n_det repeat column pad + n_det - 1, and any
// remaining column (odd n_det) is zero.  Float operations in the reference's
// order without contraction, so the result equals its float arithmetic.
// kStaged: the input row is first copied to shared memory in one coalesced pass
// (16-byte loads where the row is 16-byte aligned), so the two taps of every
// output read shared memory; rows longer than kShiftStageMax read their taps
// from global memory.  Outputs are written strided by the block size (each warp
// store one contiguous 128-byte run).
constexpr int kShiftStageMax = 12288;  // 48 KB of dynamic shared memory

template <bool kStaged>
__global__ void __launch_bounds__(kPrepThreads) shift_pad_kernel(
    const float* in, const float* xoff, float* out, int n_det, int n_ang, int out_width) {
  extern __shared__ float srow[];
  const int i = blockIdx.x, s = blockIdx.y;
  const float* r = in + ((size_t)s * n_ang + i) * n_det;
  float* o = out + ((size_t)s * n_ang + i) * out_width;
  const float x0 = xoff[s];
  const int pad = n_det / 2;
  if (kStaged) {
    int q0 = 0;
    if ((reinterpret_cast<uintptr_t>(r) & 15) == 0) {
      const int n4 = n_det >> 2;
      for (int q = threadIdx.x; q < n4; q += blockDim.x)
        reinterpret_cast<float4*>(srow)[q] = __ldg(reinterpret_cast<const float4*>(r) + q);
      q0 = 4 * n4;
    }
    for (int q = q0 + threadIdx.x; q < n_det; q += blockDim.x) srow[q] = __ldg(&r[q]);
    __syncthreads();
  }
  // Integer-valued floats below 2^24 are exact, so (float)k is kept as a float
  // counter clamped in float, and (float)nk, (float)(nk + 1) are floor(kk) and
  // floor(kk) + 1 (the sum rounds like the int-to-float conversion of nk + 1):
  // the same bits as the reference's expressions with two conversions per output
  // instead of five (the conversion pipe bounded this kernel).
  const int lim = 2 * pad + n_det;
  const float fmax_k = (float)(n_det - 1), fstep = (float)blockDim.x;
  float fkm = (float)((int)threadIdx.x - pad);  // (float)(kp - pad)
#pragma unroll 4
  for (int kp = threadIdx.x; kp < out_width; kp += blockDim.x, fkm += fstep) {
    if (kp >= lim) {
      o[kp] = 0.f;
      continue;
    }
    const float fk = fminf(fmaxf(fkm, 0.f), fmax_k);  // (float)min(max(kp - pad, 0), n_det - 1)
    const float kk = __fsub_rn(fk, x0);
    const float fl = floorf(kk);
    const int nk = (int)fl;
    const int a = min(max(nk, 0), n_det - 1);
    const int b = min(max(nk + 1, 0), n_det - 1);
    const float wa = __fsub_rn(__fadd_rn(fl, 1.f), kk);
    const float wb = __fsub_rn(kk, fl);
    const float va = kStaged ? srow[a] : __ldg(&r[a]);
    const float vb = kStaged ? srow[b] : __ldg(&r[b]);
    o[kp] = __fadd_rn(__fmul_rn(va, wa), __fmul_rn(vb, wb));
  }
}

// One block per (row, output slice); the staged form when the row fits.  128
// threads: blocks alternate between staging a row and writing it, and more
// blocks per SM overlap those phases better (16 x 2048 x 1500 to 4096-wide rows,
// us per slice: 256 threads 11.2, 128 threads 9.9, 64 threads 10.9).
constexpr int kShiftThreads = 128;

void launch_shift_pad(int n_ang, int n_slices, cudaStream_t st, const float* in, const float* xoff,
                      float* out, int n_det, int out_width) {
  const dim3 grid(n_ang, n_slices);
  if (n_det <= kShiftStageMax)
    shift_pad_kernel<true><<<grid, kShiftThreads, (size_t)n_det * sizeof(float), st>>>(
        in, xoff, out, n_det, n_ang, out_width);
  else
    shift_pad_kernel<false><<<grid, kShiftThreads, 0, st>>>(in, xoff, out, n_det, n_ang, out_width);
}

// ---------------------------------------------------------------------------
// Window copy rows [offset, offset + n) x cols [offset, offset + n); with
// radius > 0, pixels with (k - n/2)^2 + (j - n/2)^2 >= radius^2 become 0.
__global__ void crop_kernel(const float* rec, long rec_stride, long rec_slice, float* out,
                            long out_stride, long out_slice, int n, int offset, int radius) {
  const int j = blockIdx.x, s = blockIdx.y;
  const float* src = rec + (size_t)s * rec_slice + (size_t)(j + offset) * rec_stride + offset;
  float* dst = out + (size_t)s * out_slice + (size_t)j * out_stride;
  const long long r2 = (long long)radius * radius;
  const int h = n / 2;
  const long long dj = (long long)(j - h) * (j - h);
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    float v = src[k];
    if (radius > 0 && (long long)(k - h) * (k - h) + dj >= r2) v = 0.f;
    dst[k] = v;
  }
}

// ---------------------------------------------------------------------------
// Output thresholds and 8-bit slices of the reference's BMP/TIFF writer
// (gridrec/GPU/tomo_recon.cpp:2282-2361).  lo / hi: min / max over every pixel
// of the given slices (start 1e10 / -1e10; NaN compares false and is skipped),
// then capped by the configured upper / raised to the configured lower value.
// Min and max do not depend on the order of evaluation, so the block partials
// give the reference's values exactly.
constexpr int kMinMaxBlocks = 1024;

__global__ void __launch_bounds__(kPrepThreads) minmax_partial_kernel(
    const float* img, int n_slices, int rows, int cols, long row_stride, long slice_stride,
    float2* part) {
  float lo = 1e10f, hi = -1e10f;
  const long per_slice = (long)rows * cols;
  const long total = per_slice * n_slices;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long)gridDim.x * blockDim.x) {
    const long s = i / per_slice, r = (i - s * per_slice) / cols;
    const long c = i - s * per_slice - r * cols;
    const float p = img[s * slice_stride + r * row_stride + c];
    if (hi < p) hi = p;
    if (lo > p) lo = p;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
    lo = fminf(lo, l2);
    hi = fmaxf(hi, h2);
  }
  __shared__ float2 s_part[kPrepThreads / 32];
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kPrepThreads / 32; ++w) {
      lo = fminf(lo, s_part[w].x);
      hi = fmaxf(hi, s_part[w].y);
    }
    part[blockIdx.x] = make_float2(lo, hi);
  }
}

__global__ void minmax_final_kernel(const float2* part, int n, float lower_clamp, float upper_clamp,
                                    float* lohi) {
  float lo = 1e10f, hi = -1e10f;
  for (int i = 0; i < n; ++i) {
    lo = fminf(lo, part[i].x);
    hi = fmaxf(hi, part[i].y);
  }
  if (hi > upper_clamp) hi = upper_clamp;
  if (lo < lower_clamp) lo = lower_clamp;
  lohi[0] = lo;
  lohi[1] = hi;
}

// 0 below lo, 255 above hi, else (unsigned char)(255 * (p - lo) / (hi - lo)) in
// float left to right (a NaN value, which the reference's cast leaves undefined,
// gives 0); with radius > 0, pixels with (x - cols/2)^2 + (y - rows/2)^2 > radius^2
// are 0 (the writer's cropped copy keeps the boundary, unlike crop_kernel).
__global__ void to_u8_kernel(const float* img, int cols, int rows, long row_stride,
                             long slice_stride, const float* lohi, int radius, unsigned char* out,
                             long out_row_stride, long out_slice_stride) {
  const int y = blockIdx.x, s = blockIdx.y;
  const float lo = lohi[0], hi = lohi[1];
  const float* src = img + (size_t)s * slice_stride + (size_t)y * row_stride;
  unsigned char* dst = out + (size_t)s * out_slice_stride + (size_t)y * out_row_stride;
  const long long r2 = (long long)radius * radius;
  const long long dy = (long long)(y - rows / 2) * (y - rows / 2);
  for (int x = threadIdx.x; x < cols; x += blockDim.x) {
    const float p = src[x];
    unsigned char v;
    if (p < lo) v = 0;
    else if (p > hi) v = 255;
    else {
      const float q = __fdiv_rn(__fmul_rn(255.f, __fsub_rn(p, lo)), __fsub_rn(hi, lo));
      v = (q == q) ? (unsigned char)q : 0;
    }
    if (radius > 0 && (long long)(x - cols / 2) * (x - cols / 2) + dy > r2) v = 0;
    dst[x] = v;
  }
}

// ---------------------------------------------------------------------------
// Histogram entropy of a group of image windows: nbins + 1 bins of width
// inv = (vmax - vmin) / nbins, bin = (int)((x - vmin) / inv) in float
// (truncation toward zero, values outside [0, nbins] ignored), entropy =
// -sum p log2 p with p = count / (pixels in the group).
struct Window {
  const float* base;
  long row_stride, image_stride, group_stride;
  int rows, cols, group;
};

// A block counts rows blockIdx.x, + gridDim.x, ... in a histogram of its own and adds its
// counters to the group's.  Bound by the shared-memory counters (neighbouring pixels fall
// in the same or nearby bins): 16 windows of 1024 x 1024 in 10001 bins 47 -> 43 us with one
// reciprocal for all quotients; several rows at once or 1024 threads a block do not help
// (44 to 63 us).
__global__ void hist_kernel(Window w, float vmin, float inv, int nbins, unsigned* ghist) {
  extern __shared__ unsigned hist[];
  for (int b = threadIdx.x; b <= nbins; b += blockDim.x) hist[b] = 0u;
  __syncthreads();
  const int g = blockIdx.y;
  const int total_rows = w.rows * w.group;
  const float rinv = inv >= 0x1p-40f && inv <= 0x1p40f ? __frcp_rn(inv) : 0.f;  // div_by's divisors
  for (int q = blockIdx.x; q < total_rows; q += gridDim.x) {
    const int im = q / w.rows, r = q - im * w.rows;
    const float* row = w.base + (size_t)g * w.group_stride + (size_t)im * w.image_stride +
                       (size_t)r * w.row_stride;
    for (int k = threadIdx.x; k < w.cols; k += blockDim.x) {
      const float d = __fsub_rn(row[k], vmin), m = fabsf(d);
      const float f = rinv != 0.f && m >= kDivLo && m <= 0x1p100f ? div_by(d, inv, rinv) : __fdiv_rn(d, inv);
      const int ind = (int)f;  // NaN is skipped (a host cast gives INT_MIN for it)
      if (f == f && ind >= 0 && ind <= nbins) atomicAdd(&hist[ind], 1u);
    }
  }
  __syncthreads();
  unsigned* gh = ghist + (size_t)g * (nbins + 1);
  for (int b = threadIdx.x; b <= nbins; b += blockDim.x)
    if (hist[b]) atomicAdd(&gh[b], hist[b]);
}

// One block per group, a counter per thread and pass: a chain of FP64 logarithms and
// quotients (10001 bins: 28 us with 256 threads, 12 with 1024).
constexpr int kEntropyThreads = 1024;

__global__ void __launch_bounds__(kEntropyThreads) entropy_final_kernel(const unsigned* ghist, int nbins, double n, float* out) {
  __shared__ double red[32];
  const unsigned* gh = ghist + (size_t)blockIdx.x * (nbins + 1);
  double acc = 0.0;
  for (int b = threadIdx.x; b <= nbins; b += blockDim.x)
    if (gh[b]) {
      const double p = (double)gh[b] / n;
      acc += -p * log(p) / log(2.0);
    }
  acc = block_sum_d(acc, red);
  if (threadIdx.x == 0) out[blockIdx.x] = (float)acc;
}

int launch_entropy(const Window& w, int n_groups, float vmin, float vmax, int nbins,
                   unsigned* ghist, float* out, cudaStream_t st) {
  const float inv = (vmax - vmin) / (float)nbins;
  const int smem = (nbins + 1) * (int)sizeof(unsigned);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem);
    if (e != cudaSuccess) return fail(GR_ERR_CUDA, "hist smem: %s", cudaGetErrorString(e));
  }
  cudaError_t e =
      cudaMemsetAsync(ghist, 0, (size_t)n_groups * (nbins + 1) * sizeof(unsigned), st);
  if (e != cudaSuccess) return fail(GR_ERR_CUDA, "hist memset: %s", cudaGetErrorString(e));
  const int total_rows = w.rows * w.group;
  const int bx = std::max(1, std::min(total_rows, (4 * kSMs + n_groups - 1) / n_groups));
  hist_kernel<<<dim3(bx, n_groups), 512, smem, st>>>(w, vmin, inv, nbins, ghist);
  entropy_final_kernel<<<n_groups, kEntropyThreads, 0, st>>>(ghist, nbins,
                                                 (double)w.rows * w.cols * w.group, out);
  e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "entropy: %s", cudaGetErrorString(e));
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(GR_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Carves 256-byte aligned pieces out of one scratch allocation.
struct Carve {
  size_t off = 0;
  char* base = nullptr;
  template <class T> T* take(size_t count) {
    off = (off + 255) & ~size_t(255);
    T* p = reinterpret_cast<T*>(base + off);
    off += count * sizeof(T);
    return p;
  }
};

// ---------------------------------------------------------------------------
// Rotation-axis search by cross-correlation (find_shift's brute-force path:
// data_interp + cross_correlation, find_shift/src/main/find_shift.cpp:1975-2076,
// the CPU twin of cross_correlation.cu:19-413).  For translation (tx, ty) the
// match image is sampled at (nx - tx, ny - ty) for every ROI pixel by bilinear
// interpolation over the in-image neighbours, normalised by their weight
// (0 when the weight is <= 1e-5); M_avg is the ROI mean of the samples, and
//   score = sum (T - T_avg)(M - M_avg) / (T_rms sqrt(sum (M - M_avg)^2))
// (0 when T_rms or the second sum is <= 1e-5), T_rms = sqrt(sum (T - T_avg)^2).
// All arithmetic in double, as the reference's; two passes per translation
// (mean, then centred sums), block partials summed in a fixed order.
struct XcorrArgs {
  const float* templ;   // roi_h x roi_w
  const float* match;   // height x width
  int width, height, x0, y0, roi_w, roi_h;
  double tx0, ty0, dtx, dty;
  int n_tx;
  int rows_per_block;
  double* part;         // [trans][block][2]
  const double* mavg;   // [trans] (second pass)
  const double* tavg;   // template mean
};

__device__ __forceinline__ double xcorr_sample(const XcorrArgs& a, double x, double y) {
  const double fx = floor(x), fy = floor(y);
  const int nxx = (int)fx, nyy = (int)fy;
  double pix = 0.0, wsum = 0.0;
  const double ax = (double)(nxx + 1) - x, bx = x - (double)nxx;
  const double ay = (double)(nyy + 1) - y, by = y - (double)nyy;
  const bool x0ok = nxx >= 0 && nxx < a.width, x1ok = nxx + 1 >= 0 && nxx + 1 < a.width;
  const bool y0ok = nyy >= 0 && nyy < a.height, y1ok = nyy + 1 >= 0 && nyy + 1 < a.height;
  const float* m = a.match;
  if (x0ok && y0ok) {
    pix += (double)__ldg(&m[(size_t)nyy * a.width + nxx]) * ax * ay;
    wsum += ax * ay;
  }
  if (x1ok && y0ok) {
    pix += (double)__ldg(&m[(size_t)nyy * a.width + nxx + 1]) * bx * ay;
    wsum += bx * ay;
  }
  if (x0ok && y1ok) {
    pix += (double)__ldg(&m[(size_t)(nyy + 1) * a.width + nxx]) * ax * by;
    wsum += ax * by;
  }
  if (x1ok && y1ok) {
    pix += (double)__ldg(&m[(size_t)(nyy + 1) * a.width + nxx + 1]) * bx * by;
    wsum += bx * by;
  }
  return wsum > 1e-5 ? pix / wsum : 0.0;
}

// pass 0: sum of samples; pass 1: sum (T - T_avg)(M - M_avg) and sum (M - M_avg)^2
template <int PASS>
__global__ void __launch_bounds__(256) xcorr_kernel(XcorrArgs a) {
  __shared__ double red[2][8];
  const int blk = blockIdx.x, tr = blockIdx.y;
  const double tx = a.tx0 + (tr % a.n_tx) * a.dtx;
  const double ty = a.ty0 + (tr / a.n_tx) * a.dty;
  const double mavg = PASS == 1 ? a.mavg[tr] : 0.0;
  const double tavg = PASS == 1 ? *a.tavg : 0.0;
  double s0 = 0.0, s1 = 0.0;
  const int r0 = blk * a.rows_per_block, r1 = min(a.roi_h, r0 + a.rows_per_block);
  for (int r = r0; r < r1; ++r) {
    const double y = (double)(a.y0 + r) - ty;
    for (int c = threadIdx.x; c < a.roi_w; c += blockDim.x) {
      const double m = xcorr_sample(a, (double)(a.x0 + c) - tx, y);
      if (PASS == 0) {
        s0 += m;
      } else {
        const double dm = m - mavg;
        s0 += ((double)__ldg(&a.templ[(size_t)r * a.roi_w + c]) - tavg) * dm;
        s1 += dm * dm;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = s0;
    red[1][w] = s1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      t0 += red[0][k];
      t1 += red[1][k];
    }
    double* p = a.part + ((size_t)tr * gridDim.x + blk) * 2;
    p[0] = t0;
    p[1] = t1;
  }
}

// One thread per translation sums its block partials in order.  mode 0: mean
// of the samples; mode 1: the score.
__global__ void xcorr_finish_kernel(const double* part, int nblk, int n_trans, double area,
                                    double* mavg, const double* trms, double* score, int mode) {
  const int tr = blockIdx.x * blockDim.x + threadIdx.x;
  if (tr >= n_trans) return;
  double t0 = 0.0, t1 = 0.0;
  for (int b = 0; b < nblk; ++b) {
    t0 += part[((size_t)tr * nblk + b) * 2];
    t1 += part[((size_t)tr * nblk + b) * 2 + 1];
  }
  if (mode == 0) {
    mavg[tr] = t0 / area;
  } else {
    const double r = *trms;
    score[tr] = (fabs(r) > 1e-5 && fabs(t1) > 1e-5) ? t0 / (r * sqrt(t1)) : 0.0;
  }
}

// Template mean and T_rms = sqrt(sum (T - T_avg)^2), one block, fixed order.
__global__ void __launch_bounds__(256) xcorr_template_kernel(const float* t, long n, double* out) {
  __shared__ double red[8];
  __shared__ double mean_s;
  double s = 0.0;
  for (long i = threadIdx.x; i < n; i += blockDim.x) s += (double)t[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int k = 0; k < 8; ++k) m += red[k];
    mean_s = m / (double)n;
    out[0] = mean_s;
  }
  __syncthreads();
  const double mean = mean_s;
  double q = 0.0;
  for (long i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = (double)t[i] - mean;
    q += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int k = 0; k < 8; ++k) m += red[k];
    out[1] = sqrt(m);
  }
}

}  // namespace
}  // namespace gr

namespace gr {
namespace {
template <int KPT, int RB>
void launch_ring_round(dim3 grid, cudaStream_t st, float* x, float* rm, const float* c,
                       const float* g, float* part, int n_det, int n_ang, float coeff) {
  ring_round_kernel<KPT, RB><<<grid, kPrepThreads, 0, st>>>(x, rm, c, g, part, n_det, n_ang,
                                                            kRingRows, coeff);
}

// round -1: the start pass.
template <int NT, int KV, int RB>
void launch_ring_round_vec(int round, int rows, dim3 grid, cudaStream_t st, float* x, float* rm,
                           const float* c, const float* g, const float* cs, double* part, int n_det,
                           int n_ang, float coeff, int* flags) {
  if (round < 0)
    ring_round_vec_kernel<NT, KV, RB, kStart><<<grid, NT, 0, st>>>(x, rm, c, g, cs, part, n_det, n_ang,
                                                                   rows, coeff, false, flags);
  else if (round == 0)
    ring_round_vec_kernel<NT, KV, RB, kFirst><<<grid, NT, 0, st>>>(x, rm, c, g, cs, part, n_det, n_ang,
                                                                   rows, coeff, true, flags);
  else
    ring_round_vec_kernel<NT, KV, RB, kLater><<<grid, NT, 0, st>>>(
        x, rm, c, g, cs, part, n_det, n_ang, rows, coeff, (round & 1) == 0, flags);
}

constexpr int kRingRB = 2;  // rows at once at 2048 and 4096 columns, twice that below

// Rows per block on rows of whole 16-byte pieces: one wave of blocks over the GPU, in equal
// parts of whole row groups.
constexpr int ring_wave(int n_det) { return ring_blocks(ring_threads(n_det)) * kSMs; }
int ring_rows_vec(int n_slices, int n_det, int n_ang) {
  const long wave = ring_wave(n_det);
  const int rows = (int)(((long)n_ang * n_slices + wave - 1) / wave);
  const int parts = (n_ang + rows - 1) / rows;
  return ((n_ang + parts - 1) / parts + kRingGroup - 1) / kRingGroup * kRingGroup;
}
// The most partials that a call with up to n_slices slices of up to these sizes writes: at most
// one per row group and slice, and a slice's parts are at most its share of the widest wave,
// rounded up.
size_t ring_parts_vec(int n_slices, int n_ang) {
  const size_t groups = (size_t)n_slices * ((n_ang + kRingGroup - 1) / kRingGroup);
  return std::min(groups, (size_t)std::max(ring_wave(1), ring_wave(4096)) + n_slices);
}
}  // namespace
}  // namespace gr

using namespace gr;

extern "C" {

size_t gr_ring_workspace_bytes(int n_slices, int n_det, int n_ang) {
  if (n_slices < 1 || n_det < 1 || n_ang < 1) return 0;
  // column partials of either kind of rows, each with its flag; never less for smaller sizes
  const size_t vec = ring_parts_vec(n_slices, n_ang) * ((size_t)n_det * sizeof(double) + sizeof(int));
  const size_t scalar = (size_t)n_slices * ring_chunks(n_ang) * n_det * sizeof(float);
  const size_t means = (size_t)n_slices * ((size_t)n_ang + n_det + 2) * sizeof(float);
  return std::max(vec, scalar) + means + 16;
}

int gr_ring_removal(float* sinos, int n_slices, int n_det, int n_ang, float ring_coeff,
                    int iterations, void* workspace, void* stream) {
  if (!sinos || !workspace) return fail(GR_ERR_ARG, "ring removal: null pointer");
  if (n_slices < 1 || n_det < 3 || n_ang < 1 || iterations < 0)
    return fail(GR_ERR_ARG, "ring removal: need n_slices >= 1, n_det >= 3, n_ang >= 1, "
                            "iterations >= 0");
  if (iterations == 0) return GR_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int bx = (n_det + kPrepThreads - 1) / kPrepThreads;
  const int cx = (n_det + 31) / 32;
  const int cthreads = 32 * kColStrides;
  const bool vec = bx <= 16 && n_det % 4 == 0 && (reinterpret_cast<uintptr_t>(sinos) & 15) == 0;
  const int rows = vec ? ring_rows_vec(n_slices, n_det, n_ang) : kRingRows;
  const int R = (n_ang + rows - 1) / rows;
  // the column partials first, on a 16-byte boundary
  void* parts = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(workspace) + 15) & ~uintptr_t(15));
  float* part = static_cast<float*>(parts);
  double* part_vec = static_cast<double*>(parts);
  float* rowmean = part + (size_t)n_slices * R * n_det * (vec ? 2 : 1);
  float* colmean = rowmean + (size_t)n_slices * n_ang;
  float* gmean = colmean + (size_t)n_slices * n_det;
  const int kpt = bx <= 1 ? 1 : bx <= 2 ? 2 : bx <= 4 ? 4 : bx <= 8 ? 8 : 16;
  const bool fused = bx <= 16;
  {
    const int ns = n_slices;
    float* x = sinos;
    float* rm = rowmean;
    float* pt = part;
    float* cm = colmean;
    float* gm = gmean;
    float* cscale = gmean + n_slices;  // this and the flags: of the vector kernels
    int* flags = reinterpret_cast<int*>(cscale + n_slices);
    auto vec_round = [&](int m) {
      const dim3 grid(R, ns);
      auto* fn = n_det <= 512    ? launch_ring_round_vec<128, 1, 2 * kRingRB>
                 : n_det <= 1024 ? launch_ring_round_vec<128, 2, 2 * kRingRB>
                 : n_det <= 2048 ? launch_ring_round_vec<128, 4, kRingRB>
                                 : launch_ring_round_vec<256, 4, kRingRB>;
      fn(m, rows, grid, st, x, rm, cm, gm, cscale, part_vec, n_det, n_ang, ring_coeff, flags);
    };
    auto vec_means = [&](const int* fl) {
      // (one slice: few blocks and many partials, 24 loads in a row with 8 strides)
      if (R > 200)
        ring_colmean_vec_kernel<16, 32><<<dim3((n_det + 15) / 16 + 1, ns), 512, 0, st>>>(
            part_vec, rm, cm, gm, cscale, n_det, n_ang, R, fl);
      else
        ring_colmean_vec_kernel<32, 8><<<dim3((n_det + 31) / 32 + 1, ns), 256, 0, st>>>(
            part_vec, rm, cm, gm, cscale, n_det, n_ang, R, fl);
    };
    if (vec) {
      vec_round(-1);
      vec_means(flags);
      ring_first_colmean_kernel<<<dim3(cx, ns), cthreads, 0, st>>>(x, rm, cm, n_det, n_ang, R, flags);
    } else {
      ring_rowmean_kernel<<<dim3(n_ang, ns), kPrepThreads, 0, st>>>(x, rm, n_det, n_ang);
      ring_colpart_kernel<<<dim3(bx, R, ns), kPrepThreads, 0, st>>>(x, rm, pt, gm, n_det, n_ang, rows);
      ring_colmean_kernel<<<dim3(cx, ns), cthreads, 0, st>>>(pt, rm, cm, gm, n_det, n_ang, R, 1);
    }
    for (int m = 0; m < iterations; ++m) {
      if (vec) {
        vec_round(m);
        if (m + 1 < iterations)
          vec_means(nullptr);
      } else if (fused) {
        const dim3 grid(R, ns);
        switch (kpt) {
          case 1: launch_ring_round<1, 4>(grid, st, x, rm, cm, gm, pt, n_det, n_ang, ring_coeff); break;
          case 2: launch_ring_round<2, 4>(grid, st, x, rm, cm, gm, pt, n_det, n_ang, ring_coeff); break;
          case 4: launch_ring_round<4, 4>(grid, st, x, rm, cm, gm, pt, n_det, n_ang, ring_coeff); break;
          case 8: launch_ring_round<8, 4>(grid, st, x, rm, cm, gm, pt, n_det, n_ang, ring_coeff); break;
          default: launch_ring_round<16, 2>(grid, st, x, rm, cm, gm, pt, n_det, n_ang, ring_coeff);
        }
        if (m + 1 < iterations)
          ring_colmean_kernel<<<dim3(cx, ns), cthreads, 0, st>>>(pt, rm, cm, gm, n_det, n_ang, R, 0);
      } else {
        // Rows wider than 4096: separate update and column passes.
        if (m > 0) {
          ring_colpart_kernel<<<dim3(bx, R, ns), kPrepThreads, 0, st>>>(x, rm, pt, gm, n_det,
                                                                        n_ang, kRingRows);
          ring_colmean_kernel<<<dim3(cx, ns), cthreads, 0, st>>>(pt, rm, cm, gm, n_det, n_ang, R, 1);
        }
        ring_update_kernel<<<dim3(n_ang, ns), kPrepThreads, 0, st>>>(x, rm, cm, gm, n_det, n_ang,
                                                                     ring_coeff);
      }
    }
  }
  return check_launch("ring removal");
}

int gr_shift_pad(const float* in, float* out, int n_slices, int n_det, int n_ang,
                 const float* xoffsets, int out_width, void* stream) {
  if (!in || !out || !xoffsets) return fail(GR_ERR_ARG, "shift/pad: null pointer");
  if (n_slices < 1 || n_det < 1 || n_ang < 1 || out_width < n_det)
    return fail(GR_ERR_ARG, "shift/pad: need n_slices, n_det, n_ang >= 1 and out_width >= n_det");
  launch_shift_pad(n_ang, n_slices, (cudaStream_t)stream, in, xoffsets, out, n_det, out_width);
  return check_launch("shift/pad");
}

int gr_crop_center(const float* recon, long recon_stride, long recon_slice_elems, float* out,
                   long out_stride, long out_slice_elems, int n_slices, int n, int offset,
                   int radius, void* stream) {
  if (!recon || !out) return fail(GR_ERR_ARG, "crop: null pointer");
  if (n_slices < 1 || n < 1 || offset < 0 || out_stride < n || recon_stride < n + offset ||
      radius < 0)
    return fail(GR_ERR_ARG, "crop: bad sizes (n=%d offset=%d recon_stride=%ld out_stride=%ld)", n,
                offset, recon_stride, out_stride);
  crop_kernel<<<dim3(n, n_slices), kPrepThreads, 0, (cudaStream_t)stream>>>(
      recon, recon_stride, recon_slice_elems, out, out_stride, out_slice_elems, n, offset, radius);
  return check_launch("crop");
}

size_t gr_threshold_workspace_bytes(void) { return kMinMaxBlocks * sizeof(float2); }

int gr_threshold_range(const float* images, int n_slices, int rows, int cols, long row_stride,
                       long slice_stride, float lower_clamp, float upper_clamp, float* lohi,
                       void* workspace, void* stream) {
  if (!images || !lohi || !workspace) return fail(GR_ERR_ARG, "threshold: null pointer");
  if (n_slices < 1 || rows < 1 || cols < 1 || row_stride < cols ||
      (n_slices > 1 && slice_stride < (long)rows * row_stride))
    return fail(GR_ERR_ARG, "threshold: bad sizes (rows=%d cols=%d row_stride=%ld)", rows, cols,
                row_stride);
  const long total = (long)n_slices * rows * cols;
  const int blocks = (int)std::min<long>(kMinMaxBlocks, (total + kPrepThreads - 1) / kPrepThreads);
  cudaStream_t st = (cudaStream_t)stream;
  float2* part = static_cast<float2*>(workspace);
  minmax_partial_kernel<<<blocks, kPrepThreads, 0, st>>>(images, n_slices, rows, cols, row_stride,
                                                         slice_stride, part);
  int rc = check_launch("threshold: min/max");
  if (rc) return rc;
  minmax_final_kernel<<<1, 1, 0, st>>>(part, blocks, lower_clamp, upper_clamp, lohi);
  return check_launch("threshold: final");
}

int gr_to_u8(const float* images, int n_slices, int rows, int cols, long row_stride,
             long slice_stride, const float* lohi, int radius, unsigned char* out,
             long out_row_stride, long out_slice_stride, void* stream) {
  if (!images || !lohi || !out) return fail(GR_ERR_ARG, "to_u8: null pointer");
  if (n_slices < 1 || n_slices > 65535 || rows < 1 || cols < 1 || row_stride < cols ||
      out_row_stride < cols || radius < 0)
    return fail(GR_ERR_ARG, "to_u8: bad sizes (rows=%d cols=%d)", rows, cols);
  to_u8_kernel<<<dim3(rows, n_slices), kPrepThreads, 0, (cudaStream_t)stream>>>(
      images, cols, rows, row_stride, slice_stride, lohi, radius, out, out_row_stride,
      out_slice_stride);
  return check_launch("to_u8");
}

size_t gr_entropy_workspace_bytes(int n_groups, int nbins) {
  if (n_groups < 1 || nbins < 1) return 0;
  return (size_t)n_groups * (nbins + 1) * sizeof(unsigned);
}

int gr_entropy(const float* images, int n_groups, int group, int rows, int cols, long row_stride,
               long image_stride, long group_stride, float vmin, float vmax, int nbins,
               float* entropies, void* workspace, void* stream) {
  if (!images || !entropies || !workspace) return fail(GR_ERR_ARG, "entropy: null pointer");
  if (n_groups < 1 || n_groups > 65535 || group < 1 || rows < 1 || cols < 1 ||
      row_stride < cols || nbins < 1 || nbins > kMaxBins || !(vmax > vmin))
    return fail(GR_ERR_ARG, "entropy: bad sizes or range (nbins in [1, %d], vmax > vmin)",
                kMaxBins);
  Window w{images, row_stride, image_stride, group_stride, rows, cols, group};
  return launch_entropy(w, n_groups, vmin, vmax, nbins, static_cast<unsigned*>(workspace),
                        entropies, (cudaStream_t)stream);
}

int gr_reconstruct_padded(gr_plan* plan, const float* sinos, int n_slices, int n_det, int n_ang,
                          float xoffset, float* outs, long out_stride, void* stream) {
  int pn, pa, M0, max_pairs, dev;
  int rc = plan_shape(plan, &pn, &pa, &M0, &max_pairs, &dev);
  if (rc) return rc;
  if (!sinos || !outs) return fail(GR_ERR_ARG, "padded: null pointer");
  if (n_slices < 1 || pa != n_ang || pn < n_det + 2 * (n_det / 2) || out_stride < n_det)
    return fail(GR_ERR_ARG, "padded: plan must be %d angles and >= %d wide (is %d x %d)", n_ang,
                n_det + 2 * (n_det / 2), pa, pn);
  const int off = n_det / 2;
  if (off + n_det > M0)
    return fail(GR_ERR_ARG, "padded: crop window [%d, %d) exceeds the image size %d", off,
                off + n_det, M0);
  DeviceGuard guard(dev);
  cudaStream_t st = (cudaStream_t)stream;
  // shifted and padded as the spectra are formed; only the crop is transformed and written
  const long slice_in = (long)n_ang * n_det;
  const PaddedInput in{sinos, sinos + slice_in, 2 * slice_in, n_det, nullptr, xoffset};
  return plan_reconstruct_padded(plan, in, n_slices, outs, out_stride, {off, n_det, off, n_det}, st);
}

int gr_center_search(gr_plan* plan, const float* sino1, const float* sino2, int n_det, int n_ang,
                     const float* shifts, int n_cand, float hist_lo, float hist_hi, int nbins,
                     float* scores, int* best, float* best_images, void* stream) {
  int pn, pa, M0, max_pairs, dev;
  int rc = plan_shape(plan, &pn, &pa, &M0, &max_pairs, &dev);
  if (rc) return rc;
  if (!sino1 || !sino2 || !shifts || !scores) return fail(GR_ERR_ARG, "centre search: null pointer");
  if (n_cand < 1 || pa != n_ang || pn < n_det + 2 * (n_det / 2))
    return fail(GR_ERR_ARG, "centre search: plan must be %d angles and >= %d wide (is %d x %d)",
                n_ang, n_det + 2 * (n_det / 2), pa, pn);
  if (nbins < 1 || nbins > kMaxBins || !(hist_hi > hist_lo))
    return fail(GR_ERR_ARG, "centre search: nbins in [1, %d] and hist_hi > hist_lo", kMaxBins);
  const int off = n_det / 2;
  if (off + n_det > M0)
    return fail(GR_ERR_ARG, "centre search: crop window [%d, %d) exceeds the image size %d", off,
                off + n_det, M0);
  DeviceGuard guard(dev);
  cudaStream_t st = (cudaStream_t)stream;
  const int chunk = std::min(n_cand, max_pairs);  // candidates per batch (one pair each)
  const long slice_rec = (long)n_det * n_det;
  // The best images may still be on their way when the call returns: they are made from a copy,
  // so that the caller's rows are not read after that.
  const size_t kept = best_images ? (size_t)n_ang * n_det : 0;
  const ImageWindow win{off, n_det, off, n_det};  // the crop: only it is transformed and written
  Carve c;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) {
      if ((rc = plan_scratch(plan, c.off + 256, (void**)&c.base))) return rc;
      c.off = 0;
    }
    c.take<float>(kept);
    c.take<float>(kept);
    c.take<float>((size_t)2 * chunk * slice_rec);
    c.take<float>(n_cand);
    c.take<unsigned>((size_t)chunk * (nbins + 1));
    c.take<float>(n_cand);
  }
  c.off = 0;
  float* kept1 = c.take<float>(kept);
  float* kept2 = c.take<float>(kept);
  float* rec = c.take<float>((size_t)2 * chunk * slice_rec);
  float* xo = c.take<float>(n_cand);
  unsigned* gh = c.take<unsigned>((size_t)chunk * (nbins + 1));
  float* sc = c.take<float>(n_cand);
  cudaError_t e = cudaMemcpyAsync(xo, shifts, n_cand * sizeof(float), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && kept)
    e = cudaMemcpyAsync(kept1, sino1, kept * sizeof(float), cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess && kept)
    e = cudaMemcpyAsync(kept2, sino2, kept * sizeof(float), cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) return cuda_fail(e, "centre search: copies");
  for (int c0 = 0; c0 < n_cand; c0 += chunk) {
    const int nc = std::min(chunk, n_cand - c0);
    // every pair of the chunk is the given pair of slices, with the candidate's shift
    const PaddedInput in{sino1, sino2, 0, n_det, xo + c0, 0.f};
    if ((rc = plan_reconstruct_padded(plan, in, 2 * nc, rec, n_det, win, st))) return rc;
    Window w{rec, n_det, slice_rec, 2 * slice_rec, n_det, n_det, 2};
    if ((rc = launch_entropy(w, nc, hist_lo, hist_hi, nbins, gh, sc + c0, st))) return rc;
  }
  e = cudaMemcpyAsync(scores, sc, n_cand * sizeof(float), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "centre search: scores");
  // First strict minimum, as the reference's `entropy_cur < entropy_optim` scan.
  int bi = 0;
  for (int k = 1; k < n_cand; ++k)
    if (scores[k] < scores[bi]) bi = k;
  if (best) *best = bi;
  if (best_images) {
    const PaddedInput in{kept1, kept2, 0, n_det, xo + bi, 0.f};
    if ((rc = plan_reconstruct_padded(plan, in, 2, best_images, n_det, win, st))) return rc;
  }
  return GR_OK;
}

int gr_xcorr_scores(const float* templ_roi, const float* match, int width, int height, int roi_x0,
                    int roi_x1, int roi_y0, int roi_y1, double tx0, double ty0, double dtx,
                    double dty, int n_tx, int n_ty, double* scores, void* stream) {
  if (!templ_roi || !match || !scores) return fail(GR_ERR_ARG, "xcorr: null pointer");
  if (width < 1 || height < 1 || n_tx < 1 || n_ty < 1 || roi_x0 < 0 || roi_y0 < 0 ||
      roi_x1 < roi_x0 || roi_y1 < roi_y0 || roi_x1 >= width || roi_y1 >= height)
    return fail(GR_ERR_ARG, "xcorr: bad image, ROI or translation grid");
  if ((long)n_tx * n_ty > 65535) return fail(GR_ERR_ARG, "xcorr: at most 65535 translations");
  cudaStream_t st = (cudaStream_t)stream;
  const int roi_w = roi_x1 - roi_x0 + 1, roi_h = roi_y1 - roi_y0 + 1;
  const int n_trans = n_tx * n_ty;
  // enough blocks to fill the GPU: split the ROI rows when translations are few
  const int want_blocks = 4 * kSMs;
  int nblk = std::max(1, std::min(roi_h, (want_blocks + n_trans - 1) / n_trans));
  const int rows_per = (roi_h + nblk - 1) / nblk;
  nblk = (roi_h + rows_per - 1) / rows_per;
  double* d = nullptr;
  const size_t nd = (size_t)n_trans * nblk * 2 + n_trans * 2 + 2;
  cudaError_t e = cudaMallocAsync(&d, nd * sizeof(double), st);
  if (e != cudaSuccess) return fail(GR_ERR_NOMEM, "xcorr: %s", cudaGetErrorString(e));
  double* part = d;
  double* mavg = part + (size_t)n_trans * nblk * 2;
  double* sc = mavg + n_trans;
  double* tstat = sc + n_trans;  // T_avg, T_rms
  XcorrArgs a{templ_roi, match, width, height, roi_x0, roi_y0, roi_w, roi_h,
              tx0, ty0, dtx, dty, n_tx, rows_per, part, mavg, tstat};
  const int fin = (n_trans + 255) / 256;
  xcorr_template_kernel<<<1, 256, 0, st>>>(templ_roi, (long)roi_w * roi_h, tstat);
  xcorr_kernel<0><<<dim3(nblk, n_trans), 256, 0, st>>>(a);
  xcorr_finish_kernel<<<fin, 256, 0, st>>>(part, nblk, n_trans, (double)roi_w * roi_h, mavg,
                                           tstat + 1, sc, 0);
  xcorr_kernel<1><<<dim3(nblk, n_trans), 256, 0, st>>>(a);
  xcorr_finish_kernel<<<fin, 256, 0, st>>>(part, nblk, n_trans, (double)roi_w * roi_h, mavg,
                                           tstat + 1, sc, 1);
  e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(scores, sc, n_trans * sizeof(double), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(d, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? GR_OK : cuda_fail(e, "xcorr");
}

}  // extern "C"
