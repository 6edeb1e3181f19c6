// Learned correction for narrow-kernel gridrec: a 3-layer, 16-channel, 3x3
// residual CNN on the reconstructed slice,
//   h1 = relu(conv1(x)), h2 = relu(conv2(h1)), y = x + conv3(h2),
// conv1: 1 -> 16, conv2: 16 -> 16, conv3: 16 -> 1, zero padding, biases.
// Hidden activations are stored in BF16, channels last (16 per pixel); every
// sum accumulates in FP32.  conv2 -- 2304 of the 2592 multiply-adds per pixel --
// runs on the tensor cores (mma.sync m16n8k16, BF16 in, FP32 accumulate), in the
// forward pass and, with flipped and transposed weights, for the gradient with
// respect to its input, and so do the weight gradients (contractions over all pixels);
// the thin 1 -> 16 and 16 -> 1 layers run on the CUDA cores.  Partial sums are added in
// a fixed order, so training is deterministic.
//
// Parameters: one float32 array of kCnnParams entries:
//   w1[tap][co] (144), b1 (16), w2[tap][co][ci] (2304), b2 (16), w3[tap][ci] (144), b3 (1)
// with tap = (dy + 1) * 3 + (dx + 1) and conv(x)[p] = b + sum_tap w[tap] x[p + (dy, dx)].
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "gr_device.cuh"
#include "gr_internal.h"

namespace gr {
namespace {

constexpr int kC = 16;
constexpr int kW1 = 0, kB1 = 144, kW2 = 160, kB2 = 2464, kW3 = 2480, kB3 = 2624;
constexpr int kCnnParams = 2625;

__device__ __forceinline__ int tap_dy(int tap) { return tap / 3 - 1; }
__device__ __forceinline__ int tap_dx(int tap) { return tap % 3 - 1; }

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(unsigned u) {
  const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

// Pixels per thread of the thin layers (rows, or columns in conv3): the weights' 16-byte
// shared-memory reads, which bound them, serve that many pixels.
constexpr int kThinPx = 2;

// ---------------------------------------------------------------- conv1 (1 -> 16)
// Thread: pixels (xi, yi) .. (xi, yi + kThinPx - 1).
__global__ void __launch_bounds__(128) cnn_conv1_kernel(const float* params, const float* x,
                                                        __nv_bfloat16* h1, int h, int w) {
  __shared__ __align__(16) float sp[kB1 + kC];  // w1, b1
  for (int i = threadIdx.x; i < kB1 + kC; i += blockDim.x) sp[i] = params[i];
  __syncthreads();
  const int xi = blockIdx.x * blockDim.x + threadIdx.x, yi = blockIdx.y * kThinPx, im = blockIdx.z;
  if (xi >= w) return;
  const float* xm = x + (size_t)im * h * w;
  float in[kThinPx + 2][3];
#pragma unroll
  for (int r = 0; r < kThinPx + 2; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int yy = yi + r - 1, xx = xi + c - 1;
      in[r][c] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? xm[(size_t)yy * w + xx] : 0.f;
    }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    unsigned o[kThinPx][4];
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
      float4 z[kThinPx];
#pragma unroll
      for (int p = 0; p < kThinPx; ++p) z[p] = *reinterpret_cast<const float4*>(sp + kB1 + half * 8 + c);
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const float4 wt = *reinterpret_cast<const float4*>(sp + kW1 + tap * kC + half * 8 + c);
#pragma unroll
        for (int p = 0; p < kThinPx; ++p) {
          const float v = in[p + tap / 3][tap % 3];
          z[p].x = fmaf(wt.x, v, z[p].x);
          z[p].y = fmaf(wt.y, v, z[p].y);
          z[p].z = fmaf(wt.z, v, z[p].z);
          z[p].w = fmaf(wt.w, v, z[p].w);
        }
      }
#pragma unroll
      for (int p = 0; p < kThinPx; ++p) {
        o[p][c / 2] = pack_bf16(fmaxf(z[p].x, 0.f), fmaxf(z[p].y, 0.f));
        o[p][c / 2 + 1] = pack_bf16(fmaxf(z[p].z, 0.f), fmaxf(z[p].w, 0.f));
      }
    }
#pragma unroll
    for (int p = 0; p < kThinPx; ++p)
      if (yi + p < h)
        reinterpret_cast<uint4*>(h1 + (((size_t)im * h + yi + p) * w + xi) * kC)[half] =
            make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
  }
}

// ---------------------------------------------------------------- conv2 (16 -> 16), tensor cores
// One warp step: 16 consecutive pixels of a row (the M = 16 rows of the mma) x 16
// output channels (two n = 8 tiles); K = 16 input channels per tap, 9 taps.
// Fragments of mma.m16n8k16 (g = lane / 4, t = lane % 4): A rows g, g + 8 and
// columns 2t, 2t + 1, 2t + 8, 2t + 9 (pixel, input channel); B rows (input
// channels) 2t, 2t + 1, 2t + 8, 2t + 9 of column g (output channel); D rows g,
// g + 8, columns 2t, 2t + 1.
// backward = 0: out = relu(conv2(in) + b2).  backward = 1: the gradient with
// respect to conv2's input, conv with w'[tap][ci][co] = w2[8 - tap][co][ci]
// (no bias), times (mask > 0) -- the ReLU of h1.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A block of 4 warps walks down a strip of kStW columns, 16 pixels of the row per warp: the
// three input rows in use lie in a ring in shared memory (pixels kStPx bytes apart, so that
// the eight 16-byte rows of an ldmatrix fall on distinct banks), filled by cp.async a row
// ahead, so an input pixel is read once per strip instead of once per tap.  The output
// goes through shared memory to whole 16-byte stores.  4 x 1024 x 1024: 99 us
// forward or backward (201 us with A fragments loaded from global memory, 4 bytes a lane).
constexpr int kStW = 64, kStThreads = 128, kStBlocks = 4;  // blocks per SM
constexpr int kStPx = 48;                                  // bytes between pixels in shared memory
constexpr int kStHalo = kStW + 2;
struct Conv2Smem {
  alignas(16) unsigned char in[4][kStHalo * kStPx];        // ring over rows y - 1 .. y + 2
  alignas(16) unsigned char mask[2][kStW * kStPx];
  alignas(16) unsigned char out[kStW * kStPx];
};

// Segments of a strip, so that `per_sm` blocks per SM fill the GPU about once.
int strip_segments(int n_img, int h, int w, int per_sm) {
  const long strips = (long)n_img * ((w + kStW - 1) / kStW);
  return (int)std::max(1L, std::min<long>(h, (long)per_sm * kSMs / strips));
}

__device__ __forceinline__ void cp_async_zfill16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}

__global__ void __launch_bounds__(kStThreads, kStBlocks) cnn_conv2_kernel(
    const float* params, const __nv_bfloat16* in, const __nv_bfloat16* mask, __nv_bfloat16* out,
    int h, int w, int backward, int segs) {
  __shared__ Conv2Smem sm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int strip = blockIdx.x / segs, seg = blockIdx.x - strip * segs, im = blockIdx.y;
  const int x0 = strip * kStW;
  const int y0 = (int)((long)h * seg / segs), y1 = (int)((long)h * (seg + 1) / segs);
  const size_t img = (size_t)im * h * w;
  auto load_in = [&](int y) {
    const bool row = y >= 0 && y < h;
    for (int i = tid; i < 2 * kStHalo; i += kStThreads) {
      const int c = i >> 1, xx = x0 + c - 1;
      const bool ok = row && xx >= 0 && xx < w;
      const size_t p = ok ? img + (size_t)y * w + xx : 0;
      cp_async_zfill16(sm.in[y & 3] + c * kStPx + (i & 1) * 16,
                       reinterpret_cast<const unsigned char*>(in) + p * 32 + (i & 1) * 16, ok);
    }
  };
  auto load_mask = [&](int y) {
    for (int i = tid; i < 2 * kStW; i += kStThreads) {
      const int c = i >> 1, xx = x0 + c;
      const bool ok = y < h && xx < w;
      const size_t p = (ok ? img + (size_t)y * w + xx : 0) * 32 + (i & 1) * 16;
      cp_async_zfill16(sm.mask[y & 1] + c * kStPx + (i & 1) * 16,
                       reinterpret_cast<const unsigned char*>(mask) + p, ok);
    }
  };
  load_in(y0 - 1);
  load_in(y0);
  load_in(y0 + 1);
  if (mask) load_mask(y0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  // this lane's B fragments (packed BF16 pairs) of all taps and both output-channel tiles
  unsigned wb[9][2][2];
  float bias[2][2];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int n = nt * 8 + g;  // output channel
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int k = 2 * t + 8 * half;  // input channels k, k + 1
        const float* p0 = params + kW2 + (backward ? ((8 - tap) * kC + k) * kC + n : (tap * kC + n) * kC + k);
        wb[tap][nt][half] = pack_bf16(__ldg(p0), __ldg(p0 + (backward ? kC : 1)));
      }
#pragma unroll
    for (int e = 0; e < 2; ++e) bias[nt][e] = backward ? 0.f : __ldg(&params[kB2 + nt * 8 + 2 * t + e]);
  }
  const int q0 = warp * 16;
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 16;
  for (int y = y0; y < y1; ++y) {
    if (y + 1 < y1) {
      load_in(y + 2);
      if (mask) load_mask(y + 1);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // row y and its neighbours are there for every thread
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      unsigned a[4];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                   : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                   : "r"(smem_u32(sm.in[(y + tap_dy(tap)) & 3] + (q0 + 1 + tap_dx(tap) + lrow) * kStPx + lcol))
                   : "memory");
      mma_bf16(acc[0], a, wb[tap][0][0], wb[tap][0][1]);
      mma_bf16(acc[1], a, wb[tap][1][0], wb[tap][1][1]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int o = (q0 + g + 8 * half) * kStPx + (nt * 8 + 2 * t) * 2;
        float z0 = acc[nt][2 * half], z1 = acc[nt][2 * half + 1];
        if (!backward) {
          z0 = fmaxf(z0 + bias[nt][0], 0.f);
          z1 = fmaxf(z1 + bias[nt][1], 0.f);
        } else {
          const float2 m = unpack_bf16(*reinterpret_cast<const unsigned*>(sm.mask[y & 1] + o));
          z0 = m.x > 0.f ? z0 : 0.f;
          z1 = m.y > 0.f ? z1 : 0.f;
        }
        *reinterpret_cast<unsigned*>(sm.out + o) = pack_bf16(z0, z1);
      }
    __syncwarp();
    {
      const int c = q0 + (lane >> 1), xx = x0 + c;
      if (xx < w)
        *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(out) +
                                  (img + (size_t)y * w + xx) * 32 + (lane & 1) * 16) =
            *reinterpret_cast<const uint4*>(sm.out + c * kStPx + (lane & 1) * 16);
    }
    __syncthreads();  // the ring's oldest row is read before it is refilled
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// ---------------------------------------------------------------- conv3 (16 -> 1) + residual
// A thread walks down kConv3Rows rows of kThinPx columns, 128 apart, with the sums of
// three output rows of each: a loaded pixel of h2 serves three taps (6 instead of 18
// 16-byte loads per output) and a weight all columns.  Each sum takes its taps in order
// 0..8 (rows y - 1, y, y + 1).  L1-bound (16-byte loads 32 bytes apart and the weights'
// broadcasts).
constexpr int kConv3Rows = 16;

__global__ void __launch_bounds__(128) cnn_conv3_kernel(const float* params, const float* x,
                                                        const __nv_bfloat16* h2, float* y, int h,
                                                        int w) {
  __shared__ __align__(16) float sp[9 * kC + 1];  // w3, b3
  for (int i = threadIdx.x; i < 9 * kC + 1; i += blockDim.x) sp[i] = params[kW3 + i];
  __syncthreads();
  const int xi = blockIdx.x * (128 * kThinPx) + threadIdx.x, im = blockIdx.z;
  if (xi >= w) return;
  const uint4* h128 = reinterpret_cast<const uint4*>(h2) + (size_t)im * h * w * 2;
  const int y0 = blockIdx.y * kConv3Rows, y1 = min(h, y0 + kConv3Rows);
  const float bias = sp[9 * kC];
  float zp[kThinPx], zc[kThinPx], zn[kThinPx];  // output rows r - 1, r, r + 1
#pragma unroll
  for (int p = 0; p < kThinPx; ++p) zp[p] = zc[p] = zn[p] = bias;
  for (int r = y0 - 1; r <= y1; ++r) {
    if (r >= 0 && r < h) {
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        uint4 q[kThinPx][2];
#pragma unroll
        for (int p = 0; p < kThinPx; ++p) {
          const int xx = xi + 128 * p + dx - 1;
          const bool ok = xx >= 0 && xx < w;
          const uint4* s = h128 + ((size_t)r * w + (ok ? xx : 0)) * 2;
          q[p][0] = ok ? __ldg(&s[0]) : make_uint4(0u, 0u, 0u, 0u);
          q[p][1] = ok ? __ldg(&s[1]) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int c = 0; c < kC; c += 4) {
          const float4 w0 = *reinterpret_cast<const float4*>(sp + dx * kC + c);
          const float4 w1 = *reinterpret_cast<const float4*>(sp + (3 + dx) * kC + c);
          const float4 w2 = *reinterpret_cast<const float4*>(sp + (6 + dx) * kC + c);
#pragma unroll
          for (int p = 0; p < kThinPx; ++p) {
            const uint4 u = q[p][c / 8];
            const float2 v = unpack_bf16((c & 4) ? u.z : u.x), v2 = unpack_bf16((c & 4) ? u.w : u.y);
            zn[p] = fmaf(w0.w, v2.y, fmaf(w0.z, v2.x, fmaf(w0.y, v.y, fmaf(w0.x, v.x, zn[p]))));
            zc[p] = fmaf(w1.w, v2.y, fmaf(w1.z, v2.x, fmaf(w1.y, v.y, fmaf(w1.x, v.x, zc[p]))));
            zp[p] = fmaf(w2.w, v2.y, fmaf(w2.z, v2.x, fmaf(w2.y, v.y, fmaf(w2.x, v.x, zp[p]))));
          }
        }
      }
    }
#pragma unroll
    for (int p = 0; p < kThinPx; ++p) {
      if (r - 1 >= y0 && xi + 128 * p < w) {
        const size_t o = ((size_t)im * h + r - 1) * w + xi + 128 * p;
        y[o] = x[o] + zp[p];
      }
      zp[p] = zc[p];
      zc[p] = zn[p];
      zn[p] = bias;
    }
  }
}

// ---------------------------------------------------------------- backward pieces
// loss = mean (y - target)^2; gy = 2 (y - target) / N; per-block loss partials.
__global__ void cnn_loss_kernel(const float* y, const float* target, float* gy, double* part,
                                long n) {
  __shared__ double red[8];
  double s = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float d = y[i] - target[i];
    gy[i] = 2.f * d / (float)n;
    s += (double)d * d;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    part[blockIdx.x] = t;
  }
}

// g_z2[p][c] = (h2[p][c] > 0) * sum_tap w3[tap][c] gy[p - (dy, dx)]
__global__ void cnn_conv3_bwd_kernel(const float* params, const float* gy,
                                     const __nv_bfloat16* h2, __nv_bfloat16* gz2, int h, int w) {
  __shared__ __align__(16) float sp[9 * kC];  // w3
  for (int i = threadIdx.x; i < 9 * kC; i += blockDim.x) sp[i] = params[kW3 + i];
  __syncthreads();
  const int xi = blockIdx.x * blockDim.x + threadIdx.x, yi = blockIdx.y * kThinPx, im = blockIdx.z;
  if (xi >= w) return;
  const float* gm = gy + (size_t)im * h * w;
  float gin[kThinPx + 2][3];  // gy around the thread's pixels
#pragma unroll
  for (int r = 0; r < kThinPx + 2; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int yy = yi + r - 1, xx = xi + c - 1;
      gin[r][c] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? gm[(size_t)yy * w + xx] : 0.f;
    }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    unsigned mu[kThinPx][4], o[kThinPx][4];
#pragma unroll
    for (int p = 0; p < kThinPx; ++p) {
      const size_t px = ((size_t)im * h + min(yi + p, h - 1)) * w + xi;
      const uint4 mq = __ldg(reinterpret_cast<const uint4*>(h2) + px * 2 + half);
      mu[p][0] = mq.x;
      mu[p][1] = mq.y;
      mu[p][2] = mq.z;
      mu[p][3] = mq.w;
    }
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
      float4 z[kThinPx];
#pragma unroll
      for (int p = 0; p < kThinPx; ++p) z[p] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const float4 wt = *reinterpret_cast<const float4*>(sp + tap * kC + half * 8 + c);
#pragma unroll
        for (int p = 0; p < kThinPx; ++p) {
          const float v = gin[p + 2 - tap / 3][2 - tap % 3];  // gy[p - (dy, dx)]
          z[p].x = fmaf(wt.x, v, z[p].x);
          z[p].y = fmaf(wt.y, v, z[p].y);
          z[p].z = fmaf(wt.z, v, z[p].z);
          z[p].w = fmaf(wt.w, v, z[p].w);
        }
      }
#pragma unroll
      for (int p = 0; p < kThinPx; ++p) {
        const float2 m0 = unpack_bf16(mu[p][c / 2]), m1 = unpack_bf16(mu[p][c / 2 + 1]);
        o[p][c / 2] = pack_bf16(m0.x > 0.f ? z[p].x : 0.f, m0.y > 0.f ? z[p].y : 0.f);
        o[p][c / 2 + 1] = pack_bf16(m1.x > 0.f ? z[p].z : 0.f, m1.y > 0.f ? z[p].w : 0.f);
      }
    }
#pragma unroll
    for (int p = 0; p < kThinPx; ++p)
      if (yi + p < h)
        reinterpret_cast<uint4*>(gz2)[(((size_t)im * h + yi + p) * w + xi) * 2 + half] =
            make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
  }
}

// Weight gradients of all three layers on the tensor cores, contracted over pixels.
// A block of 4 warps walks down a strip of kWgW columns, 64 pixels of a row in four groups
// q of 16 (mma.m16n8k16, K = the 16 pixels):
//   dW2[tap][co][ci] = sum_q gz2[q][co] h1[q + off][ci]   A = gz2^T, B = h1 shifted
//   dW1[tap][co]     = sum_q gz1[q][co] x[q + off]         A = gz1^T, B = x's taps and a one
//   dW3[tap][ci]     = sum_q gy[q - off] h2[q][ci]         A = gy's taps, B = h2
//   db2[co] = sum gz2, db1 (the column of ones of dW1's B), db3 = sum gy
// gz1, gz2, h1 and h2 are BF16 already, so their products are exact; the FP32 operands x
// and gy enter as three BF16 parts each, which add up to the FP32 value.
// The tensor core cuts off what its FP32 accumulator cannot hold instead of rounding, so
// a sum kept in the accumulator loses up to 2^-24 of itself with every MMA (7e-6 of the
// gradients at 4 x 1024 x 1024, 6e-5 at 4096 x 4096).  Every MMA therefore starts from zero;
// its 16 pixels are added to a sum in registers (rounded to nearest), and those sums of at
// most 128 additions to FP64 sums in shared memory every kWgFlush rows.  A warp takes two
// taps of dW2 for the whole row, and tap 8, dW1, dW3 and the biases for its own group of 16
// pixels, so that its sums fit the registers.
// Rows arrive by cp.async a row ahead into rings (three rows of h1, x and gy are in use);
// pixels lie 48 bytes apart, so that the eight 16-byte rows of an ldmatrix fall on distinct
// banks.
// Bound: the latency of a row's exchanges (one row of 64 pixels per barrier), then DRAM
// (136 bytes per pixel).  4 x 1024 x 1024: 247 us and 6 us for the reduction of 384 blocks,
// error against the exact contraction of the same operands 2.4e-8 to 2.9e-8; 237 us and
// up to 8e-6 with the sums kept in the accumulators; 2179 us on the CUDA cores and 1444 us for the
// reduction of 32768 segments, 2.4e-8 to 2.9e-8.
constexpr int kWgW = kStW, kWgThreads = 128, kWgBlocks = 3;  // blocks per SM
constexpr int kWgFlush = 32;                                 // rows: 4 additions each
constexpr int kWgPx = kStPx;
constexpr int kWgHalo = kWgW + 2;
// A warp's FP64 sums: dW2 of its two taps and of tap 8, then those of its own pixels.
constexpr int kWgOwn = 3 * kC * kC;  // dW1, db1, dW3, db2, db3
constexpr int kWgOwnB1 = kWgOwn + 9 * kC, kWgOwnW3 = kWgOwnB1 + kC, kWgOwnB2 = kWgOwnW3 + 9 * kC;
constexpr int kWgOwnB3 = kWgOwnB2 + kC, kWgSums = kWgOwnB3 + 1;
struct WgSmem {
  alignas(16) unsigned char h1[4][kWgHalo * kWgPx];        // ring over rows y - 1 .. y + 2
  alignas(16) unsigned char g1[2][kWgW * kWgPx], g2[2][kWgW * kWgPx], h2[2][kWgW * kWgPx];
  float x[4][kWgHalo], gy[4][kWgHalo];
  double sums[kWgThreads / 32][kWgSums];
};

int wg_segments(int n_img, int h, int w) { return strip_segments(n_img, h, w, kWgBlocks); }
long wg_blocks(int n_img, int h, int w) {
  return (long)n_img * ((w + kWgW - 1) / kWgW) * wg_segments(n_img, h, w);
}
// The most blocks of a call of up to these sizes: wg_blocks falls where a strip more leaves
// room for fewer segments of each.
size_t wg_blocks_bound(int n_img, int h, int w) {
  const size_t strips = (size_t)n_img * ((w + kWgW - 1) / kWgW);
  return std::max(strips, std::min(strips * h, (size_t)kWgBlocks * kSMs));
}

__device__ __forceinline__ void cp_async_zfill4(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "r"(ok ? 4 : 0)
               : "memory");
}
// Four 8 x 8 BF16 blocks of 16 pixels x 16 channels at `px` (pixel stride kWgPx), transposed:
// r[0] pixels 0..7 of channels 0..7, r[1] channels 8..15, r[2], r[3] pixels 8..15 -- the
// A fragment (row = channel, column = pixel) in the order a0 a1 a2 a3, and the B fragments
// (row = pixel, column = channel) of the channel halves, (r[0], r[2]) and (r[1], r[3]).
__device__ __forceinline__ void ldm_t(unsigned (&r)[4], const unsigned char* px, int lane) {
  const unsigned char* p = px + ((lane & 7) + ((lane >> 4) & 1) * 8) * kWgPx + ((lane >> 3) & 1) * 16;
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p))
               : "memory");
}
// (a, b) as three packed BF16 pairs that sum to the FP32 values
__device__ __forceinline__ void split3(float a, float b, unsigned (&o)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    o[k] = pack_bf16(a, b);
    const float2 h = unpack_bf16(o[k]);
    a -= h.x;
    b -= h.y;
  }
}

// The MMA from zero: d = a b.
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                              unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void add4(float (&s)[4], const float (&d)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = __fadd_rn(s[i], d[i]);
}

__global__ void __launch_bounds__(kWgThreads, kWgBlocks) cnn_wgrad_kernel(
    const float* x, const float* gy, const __nv_bfloat16* h1, const __nv_bfloat16* h2,
    const __nv_bfloat16* gz1, const __nv_bfloat16* gz2, float* part, int h, int w, int segs) {
  extern __shared__ __align__(16) unsigned char smw[];
  WgSmem& sm = *reinterpret_cast<WgSmem*>(smw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int strip = blockIdx.x / segs, seg = blockIdx.x - strip * segs, im = blockIdx.y;
  const int x0 = strip * kWgW;
  const int y0 = (int)((long)h * seg / segs), y1 = (int)((long)h * (seg + 1) / segs);
  const size_t img = (size_t)im * h * w;
  // row y with a pixel of halo on both sides: h1, x and gy
  auto load_halo_row = [&](int y) {
    const int slot = y & 3;
    const bool row = y >= 0 && y < h;
    for (int i = tid; i < 2 * kWgHalo; i += kWgThreads) {
      const int c = i >> 1, xx = x0 + c - 1;
      const bool ok = row && xx >= 0 && xx < w;
      const size_t p = ok ? img + (size_t)y * w + xx : 0;
      cp_async_zfill16(sm.h1[slot] + c * kWgPx + (i & 1) * 16,
                       reinterpret_cast<const unsigned char*>(h1) + p * 32 + (i & 1) * 16, ok);
      if (i & 1) cp_async_zfill4(&sm.x[slot][c], x + p, ok);
      else cp_async_zfill4(&sm.gy[slot][c], gy + p, ok);
    }
  };
  // row y without halo: gz1, gz2 and h2
  auto load_row = [&](int y) {
    const int slot = y & 1;
    for (int i = tid; i < 2 * kWgW; i += kWgThreads) {
      const int c = i >> 1, xx = x0 + c;
      const bool ok = y < h && xx < w;
      const size_t p = (ok ? img + (size_t)y * w + xx : 0) * 32 + (i & 1) * 16;
      const int o = c * kWgPx + (i & 1) * 16;
      cp_async_zfill16(sm.g1[slot] + o, reinterpret_cast<const unsigned char*>(gz1) + p, ok);
      cp_async_zfill16(sm.g2[slot] + o, reinterpret_cast<const unsigned char*>(gz2) + p, ok);
      cp_async_zfill16(sm.h2[slot] + o, reinterpret_cast<const unsigned char*>(h2) + p, ok);
    }
  };
  // this warp's FP32 sums: dW2 of taps 2 warp, 2 warp + 1 and 8 (two n = 8 tiles each), dW1,
  // dW3, db2, db3
  float a2[3][2][4], a1[2][4], a3[2][4], ab[4], b3 = 0.f;
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int k = 0; k < 3; ++k) a2[k][n][i] = 0.f;
        a1[n][i] = a3[n][i] = 0.f;
      }
      ab[i] = 0.f;
    }
    b3 = 0.f;
  };
  clear();
  double* sums = sm.sums[warp];
  for (int i = lane; i < kWgSums; i += 32) sums[i] = 0.0;
  const unsigned one2 = lane < 4 ? 0x3f803f80u : 0u;  // B column 0 of ones
  load_halo_row(y0 - 1);
  load_halo_row(y0);
  load_halo_row(y0 + 1);
  load_row(y0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  const int g = lane >> 2, t = lane & 3;
  const int q0 = warp * 16;  // this warp's own pixels of the row
  __syncwarp();              // its sums are zero for all its lanes
  for (int y = y0; y < y1; ++y) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // row y and its neighbours are there for every thread, row y - 2 is free
    if (y + 1 < y1) {
      load_halo_row(y + 2);
      load_row(y + 1);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    unsigned fa[4], fb[4];
    float d[4], small[4];
    // dW2 of tap `tap` over the 16 pixels at q, whose gz2 fa holds
    auto tap_sums = [&](float (&s)[2][4], int tap, int q) {
      ldm_t(fb, sm.h1[(y + tap_dy(tap)) & 3] + (q + 1 + tap_dx(tap)) * kWgPx, lane);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mma_bf16_zero(d, fa, fb[n], fb[n + 2]);
        add4(s[n], d);
      }
    };
#pragma unroll
    for (int q = 0; q < kWgW; q += 16) {
      ldm_t(fa, sm.g2[y & 1] + q * kWgPx, lane);
      tap_sums(a2[0], 2 * warp, q);
      tap_sums(a2[1], 2 * warp + 1, q);
    }
    ldm_t(fa, sm.g2[y & 1] + q0 * kWgPx, lane);
    tap_sums(a2[2], 8, q0);
    mma_bf16_zero(d, fa, one2, one2);
    add4(ab, d);
    // dW1: B column n = tap (n = 9: ones); this lane's columns g and g + 8.  The two
    // small parts share an accumulator, the largest has its own.
    ldm_t(fa, sm.g1[y & 1] + q0 * kWgPx, lane);
    {
      const float* r = sm.x[(y + g / 3 - 1) & 3] + q0 + g % 3;  // x[q + off(g)], halo offset in
      unsigned lo[3], hi[3];
      split3(r[2 * t], r[2 * t + 1], lo);
      split3(r[2 * t + 8], r[2 * t + 9], hi);
      mma_bf16_zero(small, fa, lo[2], hi[2]);
      mma_bf16(small, fa, lo[1], hi[1]);
      mma_bf16_zero(d, fa, lo[0], hi[0]);
      add4(d, small);
      add4(a1[0], d);
      const float* r8 = sm.x[(y + 1) & 3] + q0 + 2;             // tap 8
      split3(r8[2 * t], r8[2 * t + 1], lo);
      split3(r8[2 * t + 8], r8[2 * t + 9], hi);
      const unsigned one = g == 1 ? 0x3f803f80u : 0u;
      mma_bf16_zero(small, fa, g == 0 ? lo[2] : 0u, g == 0 ? hi[2] : 0u);
      mma_bf16(small, fa, g == 0 ? lo[1] : 0u, g == 0 ? hi[1] : 0u);
      mma_bf16_zero(d, fa, g == 0 ? lo[0] : one, g == 0 ? hi[0] : one);
      add4(d, small);
      add4(a1[1], d);
    }
    // dW3: A row m = tap; this lane's rows g and g + 8 (tap 8 for g = 0)
    ldm_t(fb, sm.h2[y & 1] + q0 * kWgPx, lane);
    {
      const float* r = sm.gy[(y - (g / 3 - 1)) & 3] + q0 + 2 - g % 3;  // gy[q - off(g)]
      const float* r8 = sm.gy[(y - 1) & 3] + q0;                        // tap 8
      unsigned lo[3], hi[3], lo8[3], hi8[3];
      split3(r[2 * t], r[2 * t + 1], lo);
      split3(r[2 * t + 8], r[2 * t + 9], hi);
      split3(r8[2 * t], r8[2 * t + 1], lo8);
      split3(r8[2 * t + 8], r8[2 * t + 9], hi8);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int k = 2; k >= 0; --k) {
          const unsigned a[4] = {lo[k], g == 0 ? lo8[k] : 0u, hi[k], g == 0 ? hi8[k] : 0u};
          if (k == 2) mma_bf16_zero(small, a, fb[n], fb[n + 2]);
          else if (k == 1) mma_bf16(small, a, fb[n], fb[n + 2]);
          else mma_bf16_zero(d, a, fb[n], fb[n + 2]);
        }
        add4(d, small);
        add4(a3[n], d);
      }
      if (lane < 16) b3 += sm.gy[y & 3][q0 + 1 + lane];
    }
    if ((y - y0) % kWgFlush == kWgFlush - 1 || y == y1 - 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = g + (i >> 1) * 8, col = 2 * t + (i & 1);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
#pragma unroll
          for (int k = 0; k < 3; ++k) sums[(k * kC + row) * kC + n * 8 + col] += a2[k][n][i];
          const int tap1 = n * 8 + col;                      // a1: row = co, column = tap
          if (tap1 < 9) sums[kWgOwn + tap1 * kC + row] += a1[n][i];
          if (tap1 == 9) sums[kWgOwnB1 + row] += a1[n][i];
          if (row < 9) sums[kWgOwnW3 + row * kC + n * 8 + col] += a3[n][i];  // a3: row = tap, column = ci
        }
        if (col == 0) sums[kWgOwnB2 + row] += ab[i];
      }
      double s = b3;
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) sums[kWgOwnB3] += s;
      clear();
    }
  }
  __syncthreads();
  // the block's sums, those that every warp holds in warp order
  float* out = part + ((size_t)im * gridDim.x + blockIdx.x) * kCnnParams;
  auto all = [&](int i) { return (float)(((sm.sums[0][i] + sm.sums[1][i]) + sm.sums[2][i]) + sm.sums[3][i]); };
  constexpr int kTap = kC * kC;
  for (int i = tid; i < 8 * kTap; i += kWgThreads)
    out[kW2 + i] = (float)sm.sums[i / (2 * kTap)][i % (2 * kTap)];
  for (int i = tid; i < kTap; i += kWgThreads) out[kW2 + 8 * kTap + i] = all(2 * kTap + i);
  for (int i = tid; i < 9 * kC; i += kWgThreads) {
    out[kW1 + i] = all(kWgOwn + i);
    out[kW3 + i] = all(kWgOwnW3 + i);
  }
  if (tid < kC) {
    out[kB1 + tid] = all(kWgOwnB1 + tid);
    out[kB2 + tid] = all(kWgOwnB2 + tid);
  }
  if (tid == 0) out[kB3] = all(kWgOwnB3);
}

// grads[k] = sum over blocks (fixed order) of part[block][k], in double: 32 parameters x 8
// strides per block.
__global__ void __launch_bounds__(256) cnn_reduce_kernel(const float* part, long nblk, float* grads) {
  __shared__ double sums[8][32];
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), q = threadIdx.x >> 5;
  double s = 0.0;
  if (k < kCnnParams)
    for (long i = q; i < nblk; i += 8) s += part[i * kCnnParams + k];
  sums[q][threadIdx.x & 31] = s;
  __syncthreads();
  if (q == 0 && k < kCnnParams) {
    for (int i = 1; i < 8; ++i) s += sums[i][threadIdx.x & 31];
    grads[k] = (float)s;
  }
}

__global__ void cnn_adam_kernel(float* params, const float* grads, float* m, float* v, int n,
                                float lr, float b1, float b2, float eps, float c1, float c2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float g = grads[k];
  const float mk = b1 * m[k] + (1.f - b1) * g;
  const float vk = b2 * v[k] + (1.f - b2) * g * g;
  m[k] = mk;
  v[k] = vk;
  params[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
}

// ---------------------------------------------------------------- fused inference, tcgen05
// One CTA (kFThreads / 32 warps) computes output tiles of kFTh x kFTw pixels.  The tile's x region
// ((kFTh + 6) x (kFTw + 6) pixels), its h1 and h2 and conv3's per-tap partials stay in
// shared memory; only x is read from HBM and y written.  Positions of the x region are
// flattened with row stride kFWt, so a 3x3 tap (dy, dx) is the constant offset
// dy kFWt + dx: conv2 on a block of 128 consecutive positions is nine tcgen05 MMAs whose
// A operand is the same activation plane started dy kFWt + dx positions later -- no
// im2col copy.  The layers:
//  * conv1 (1 -> 16): a tcgen05 MMA per block of 128 positions on a 16-wide im2col of x
//    (the nine taps and seven zeros, BF16) built in shared memory, against w1 in BF16,
//    on the rows conv2 reads (rows 1..kFTh+4 of the x region); the im2col is dead once
//    the MMAs are done, and h1 = relu(conv1 + b1) in BF16 is written over it;
//  * conv2 (16 -> 16): tcgen05.mma kind::f16, BF16 operands from shared memory (A: 128
//    positions x 16 input channels, K-major, two 8-channel planes; B: the tap's 16 x 16
//    weights), FP32 accumulator in tensor memory (M = 128, N = 16, K = 16; one MMA per
//    tap), then bias, ReLU and BF16 on the way back to shared memory;
//  * conv3 (16 -> 1): a 1x1 tcgen05 MMA to the nine per-tap partials
//    Z[p][tap] = sum_ci w3[tap][ci] h2[p][ci] (w3 in BF16; N = 16, taps 9..15 zero), then
//    y[p] = x[p] + (b3 + sum_tap Z[p + (dy, dx)][tap]) in FP32 on the CUDA cores.  (Nine
//    shifted MMAs into one column would drop the partials, but every N = 16 MMA reads its
//    4 KB A operand from shared memory, about 30 cycles of the SM's shared-memory
//    bandwidth: eight more of them per block cost more than the partials' stores and loads.)
// Positions outside the image hold zero x, h1 and h2 (the network's zero padding); the
// wrap-around columns of the flattened rows produce values only at positions that no
// kept output reads.  One thread issues the MMAs; completion is a tcgen05.commit on an
// mbarrier with bounded waits (timeout: error word, early exit).  Each CTA holds
// kFTmemCols tensor-memory columns; its dynamic shared memory (kFSmemLaunch) admits at
// most kFCtas CTAs per SM, whose allocations fit the SM's 512 columns together, so an
// allocation never waits on another CTA.

constexpr int kFTh = 8, kFTw = 64;
constexpr int kFThreads = 128, kFCtas = 4;                     // 4 warps, 4 CTAs per SM
constexpr int kFGroups = kFThreads / 128;                      // warp groups sharing the blocks
constexpr int kFWt = kFTw + 6;                                 // flattened row stride
constexpr int kFRows = kFTh + 6;
constexpr int kFPos = kFRows * kFWt;                           // positions of the x region
constexpr int kFQ1 = kFWt, kFQ1e = (kFTh + 5) * kFWt;          // conv1: rows 1..kFTh+4
constexpr int kFQ2 = 2 * kFWt;                                 // first conv2 / conv3 position
constexpr int kFBlocks = ((kFTh + 4) * kFWt - kFQ2 + 127) / 128;  // 128-position blocks
constexpr int kFBlocks1 = (kFQ1e - kFQ1 + 127) / 128;           // conv1's blocks from kFQ1
constexpr int kFZ = 128 * kFBlocks;                            // partials per tap
constexpr int kFPlane = ((kFQ1 + 128 * kFBlocks1 > kFQ2 + kFZ + kFWt + 1 ? kFQ1 + 128 * kFBlocks1
                                                                         : kFQ2 + kFZ + kFWt + 1) +
                         127) / 128 * 128;                     // positions per activation plane
constexpr int kFXOff = 72;                                     // x buffer: reads at q - 71 .. q + 71
constexpr int kFXLen = kFPos + 2 * kFXOff;
constexpr int kFTmemNeed = 16 * (kFBlocks1 > kFBlocks ? kFBlocks1 : kFBlocks);
constexpr int kFTmemCols = kFTmemNeed <= 32 ? 32 : kFTmemNeed <= 64 ? 64 : kFTmemNeed <= 128 ? 128
                                                                                                : 256;
constexpr int kFParams = 177;                                  // w1, b1, b2, b3 in FP32
// shared memory: activation planes | B2 (9 taps) | B3 | B1 | x | FP32 params | mbarrier, tmem slot
constexpr int kFSmAct = 0, kFSmB2 = 2 * kFPlane * 16, kFSmB3 = kFSmB2 + 9 * 512;
constexpr int kFSmB1 = kFSmB3 + 512;
constexpr int kFSmX = kFSmB1 + 512, kFSmP = kFSmX + kFXLen * 4;
constexpr int kFSmBar = (kFSmP + kFParams * 4 + 15) & ~15;
constexpr int kFSmUsed = kFSmBar + 16;
constexpr int kFSmemLaunch = (228 * 1024 / kFCtas - 1024) & ~1023;
static_assert(kFQ2 + kFZ + kFWt + 1 <= kFPlane, "conv2's shifted reads stay inside the planes");
static_assert(kFQ1 + 128 * kFBlocks1 <= kFPlane, "conv1's blocks fit the planes");
static_assert(kFTmemNeed <= kFTmemCols && kFCtas * kFTmemCols <= 512,
              "accumulators fit the tensor-memory allocation, and every CTA of an SM gets one");
static_assert(9 * kFZ * 4 <= 2 * kFPlane * 16, "conv3's partials fit the activation buffer");
static_assert(kFSmUsed <= kFSmemLaunch && (kFCtas + 1) * (kFSmemLaunch + 1024) > 228 * 1024,
              "at most kFCtas CTAs per SM");

__device__ __forceinline__ uint64_t cnn_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  // start >> 4 [0,14), leading-dimension offset >> 4 [16,30), stride offset >> 4
  // [32,46), version 1 [46,48); no swizzle, base offset 0 (K-major core matrices of
  // 8 rows x 16 bytes)
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// instruction descriptor: D f32 [4,6) = 1, A bf16 [7,10) = 1, B bf16 [10,13) = 1, both
// K-major, N = 16 [17,23) = 16 >> 3, M = 128 [24,29) = 128 >> 4
constexpr uint32_t kCnnIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) |
                               ((128u >> 4) << 24);

__device__ __forceinline__ void cnn_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(da), "l"(db), "r"(kCnnIdesc), "r"(acc));
}
__device__ __forceinline__ void cnn_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// relu(v + b) of two channels in BF16 (packed FP32 add, then one converting relu)
__device__ __forceinline__ unsigned relu_bias_pack(float v0, float v1, float b0, float b1) {
  unsigned long long s;
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%1, %2};\n mov.b64 y, {%3, %4};\n"
      " add.rn.f32x2 %0, x, y;\n}" : "=l"(s) : "f"(v0), "f"(v1), "f"(b0), "f"(b1));
  unsigned r;
  asm("{\n .reg .f32 lo, hi;\n mov.b64 {lo, hi}, %1;\n cvt.rn.relu.bf16x2.f32 %0, hi, lo;\n}"
      : "=r"(r) : "l"(s));
  return r;
}
// 16 accumulator columns of this warp's 32 lanes
__device__ __forceinline__ void cnn_tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

__global__ void __launch_bounds__(kFThreads, kFCtas) cnn_fused_kernel(const float* params, const float* x,
                                                                       float* y, const float* scale,
                                                                       int n_img, int h, int w,
                                                                       int* err) {
  extern __shared__ __align__(1024) unsigned char smf[];
  uint4* act = reinterpret_cast<uint4*>(smf + kFSmAct);  // plane g: act[g kFPlane + q] = 8 BF16 channels
  unsigned short* b2s = reinterpret_cast<unsigned short*>(smf + kFSmB2);
  unsigned short* b3s = reinterpret_cast<unsigned short*>(smf + kFSmB3);
  unsigned short* b1s = reinterpret_cast<unsigned short*>(smf + kFSmB1);
  float* xs = reinterpret_cast<float*>(smf + kFSmX) + kFXOff;
  float* pw = reinterpret_cast<float*>(smf + kFSmP);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smf + kFSmBar);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smf + kFSmBar + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // B operands in BF16, K-major core matrices [ci / 8][n][ci % 8]: conv2's taps (n = co)
  // and conv3's 1x1 matrix (n = tap, taps 9..15 zero); FP32 w1, b1, b2, b3
  for (int e = tid; e < 9 * 256; e += kFThreads) {
    const int t = e >> 8, g = (e >> 7) & 1, co = (e >> 3) & 15, k8 = e & 7;
    const __nv_bfloat16 v = __float2bfloat16_rn(params[kW2 + (t * kC + co) * kC + g * 8 + k8]);
    b2s[e] = *reinterpret_cast<const unsigned short*>(&v);
  }
  for (int e = tid; e < 256; e += kFThreads) {
    const int g = e >> 7, n = (e >> 3) & 15, k8 = e & 7;
    const __nv_bfloat16 v = __float2bfloat16_rn(n < 9 ? params[kW3 + n * kC + g * 8 + k8] : 0.f);
    b3s[e] = *reinterpret_cast<const unsigned short*>(&v);
  }
  for (int e = tid; e < 256; e += kFThreads) {  // conv1: n = co, k = tap (taps 9..15 zero)
    const int g = e >> 7, co = (e >> 3) & 15, k = g * 8 + (e & 7);
    const __nv_bfloat16 v = __float2bfloat16_rn(k < 9 ? params[kW1 + k * kC + co] : 0.f);
    b1s[e] = *reinterpret_cast<const unsigned short*>(&v);
  }
  for (int i = tid; i < kFParams; i += kFThreads)
    pw[i] = i < kB1 + kC ? params[i] : (i < kB1 + 2 * kC ? params[kB2 + i - kB1 - kC] : params[kB3]);
  for (int i = tid; i < kFXLen; i += kFThreads) xs[i - kFXOff] = 0.f;
  for (int i = tid; i < 2 * kFPlane; i += kFThreads) act[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)), "n"(kFTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async();  // the B operands and zeroed planes, before the tensor core reads them
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  // descriptors: a position offset q adds q to the start-address field (16-byte units)
  const uint64_t da = cnn_smem_desc(smem_u32(act), kFPlane * 16, 128);
  const uint64_t db1 = cnn_smem_desc(smem_u32(b1s), 256, 128);
  const uint64_t db2 = cnn_smem_desc(smem_u32(b2s), 256, 128);
  const uint64_t db3 = cnn_smem_desc(smem_u32(b3s), 256, 128);
  const float b3 = pw[kB1 + 2 * kC];
  float bias1[kC], bias2[kC];
#pragma unroll
  for (int c = 0; c < kC; ++c) {
    bias1[c] = pw[kB1 + c];
    bias2[c] = pw[kB1 + kC + c];
  }
  const int tiles_x = (w + kFTw - 1) / kFTw, tiles_y = (h + kFTh - 1) / kFTh;
  const long n_tiles = (long)n_img * tiles_x * tiles_y;
  const int lq = warp & 3;  // this warp's quarter of the tensor-memory lanes
  unsigned phase = 0;
  bool ok = true;
  // the x region of a tile (zero outside the image), this thread's positions
  // tid + k kFThreads; loaded one tile ahead into registers, so that the loads' latency
  // passes during the previous tile's work
  constexpr int kXPer = (kFPos + kFThreads - 1) / kFThreads;
  float xr[kXPer], x_inv = 1.f;
  const int r_tid = tid / kFWt, c_tid = tid - r_tid * kFWt;
  auto load_x = [&](long t) {
    const int im = (int)(t / ((long)tiles_x * tiles_y));
    const int rem = (int)(t - (long)im * tiles_x * tiles_y);
    const int ty0 = (rem / tiles_x) * kFTh, tx0 = (rem % tiles_x) * kFTw;
    const bool all_in = t < n_tiles && ty0 >= 3 && tx0 >= 3 && ty0 + kFTh + 3 <= h &&
                        tx0 + kFTw + 3 <= w;
    const float* xm = x + (size_t)im * h * w;
    // the image's 1 / scale, applied when the values are stored to shared memory (a
    // product here would wait on the loads)
    x_inv = scale && t < n_tiles ? 1.f / __ldg(&scale[im]) : 1.f;
    int r = r_tid, c = c_tid;  // position tid + k kFThreads = (r, c)
#pragma unroll
    for (int k = 0; k < kXPer; ++k) {
      const int iy = ty0 - 3 + r, ix = tx0 - 3 + c;
      const bool in = tid + k * kFThreads < kFPos &&
                      (all_in || (t < n_tiles && iy >= 0 && iy < h && ix >= 0 && ix < w));
      xr[k] = in ? __ldg(&xm[(size_t)iy * w + ix]) : 0.f;
      r += kFThreads / kFWt;
      c += kFThreads % kFWt;
      if (c >= kFWt) {
        c -= kFWt;
        ++r;
      }
    }
  };
  load_x(blockIdx.x);
  for (long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int im = (int)(tile / ((long)tiles_x * tiles_y));
    const int rem = (int)(tile - (long)im * tiles_x * tiles_y);
    const int y0 = (rem / tiles_x) * kFTh, x0 = (rem % tiles_x) * kFTw;
    // a tile whose x region lies inside the image needs no zero padding
    const bool all_in = y0 >= 3 && x0 >= 3 && y0 + kFTh + 3 <= h && x0 + kFTw + 3 <= w;
    auto inside = [&](int q) {
      if (all_in) return true;
      const int r = q / kFWt, c = q - (q / kFWt) * kFWt;
      const int iy = y0 - 3 + r, ix = x0 - 3 + c;
      return iy >= 0 && iy < h && ix >= 0 && ix < w;
    };
#pragma unroll
    for (int k = 0; k < kXPer; ++k)
      if (tid + k * kFThreads < kFPos) xs[tid + k * kFThreads] = xr[k] * x_inv;
    __syncthreads();
    load_x(tile + gridDim.x);  // the next tile's x, in flight during this tile
    // conv1's im2col (BF16): plane 0 holds taps 0..7 of position q, plane 1 tap 8 and
    // zeros; conv1's blocks cover [kFQ1, kFQ1 + 128 kFBlocks1)
    for (int q = kFQ1 + tid; q < kFQ1 + 128 * kFBlocks1; q += kFThreads) {
      float in[9];
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) in[tap] = xs[q + tap_dy(tap) * kFWt + tap_dx(tap)];
      act[q] = make_uint4(pack_bf16(in[0], in[1]), pack_bf16(in[2], in[3]),
                          pack_bf16(in[4], in[5]), pack_bf16(in[6], in[7]));
      act[kFPlane + q] = make_uint4(pack_bf16(in[8], 0.f), 0u, 0u, 0u);
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int b = 0; b < kFBlocks1; ++b) cnn_mma(tmem + 16 * b, da + (kFQ1 + 128 * b), db1, 0u);
      cnn_commit(bar);
    }
    bool got = warp == 0 ? mbar_wait(bar, phase) : true;
    if (__syncthreads_or(!got)) {
      ok = false;
      break;
    }
    phase ^= 1u;
    tc_fence_after();
    // h1 = relu(conv1 + b1) in BF16 over the im2col (every MMA reading it is done); zero
    // outside the image and beyond conv1's rows; the planes' other positions are
    // cleared of the previous tile's values
    for (int b = warp >> 2; b < kFBlocks1; b += kFGroups) {
      float v[16];
      cnn_tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + 16 * b, v);
      const int q = kFQ1 + 128 * b + 32 * lq + lane;
      uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
      if (q < kFQ1e && inside(q)) {
        unsigned o[kC / 2];
#pragma unroll
        for (int c = 0; c < kC; c += 2) o[c / 2] = relu_bias_pack(v[c], v[c + 1], bias1[c], bias1[c + 1]);
        lo = make_uint4(o[0], o[1], o[2], o[3]);
        hi = make_uint4(o[4], o[5], o[6], o[7]);
      }
      act[q] = lo;
      act[kFPlane + q] = hi;
    }
    for (int i = tid; i < kFPlane - 128 * kFBlocks1; i += kFThreads) {
      const int q = i < kFQ1 ? i : i + 128 * kFBlocks1;
      act[q] = act[kFPlane + q] = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    // conv2: nine MMAs per block of 128 positions, A shifted by the tap's offset
    if (tid == 0) {
      tc_fence_after();
#pragma unroll 2
      for (int b = 0; b < kFBlocks; ++b)
#pragma unroll
        for (int t = 0; t < 9; ++t)
          cnn_mma(tmem + 16 * b, da + (kFQ2 + 128 * b + tap_dy(t) * kFWt + tap_dx(t)),
                  db2 + 32 * t, t > 0 ? 1u : 0u);
      cnn_commit(bar);
    }
    // one warp polls the barrier; the others wait at the CTA barrier (no issue slots)
    got = warp == 0 ? mbar_wait(bar, phase) : true;
    if (__syncthreads_or(!got)) {
      ok = false;
      break;
    }
    phase ^= 1u;
    tc_fence_after();
    // h2 = relu(conv2 + b2) in BF16 over h1's planes (every MMA reading h1 is done);
    // warp group g (4 warps, one per quarter of the lanes) takes blocks g, g + kFGroups, ...
    for (int b = warp >> 2; b < kFBlocks; b += kFGroups) {
      float v[16];
      cnn_tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + 16 * b, v);
      const int q = kFQ2 + 128 * b + 32 * lq + lane;
      uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
      if (inside(q)) {
        unsigned o[kC / 2];
#pragma unroll
        for (int c = 0; c < kC; c += 2) o[c / 2] = relu_bias_pack(v[c], v[c + 1], bias2[c], bias2[c + 1]);
        lo = make_uint4(o[0], o[1], o[2], o[3]);
        hi = make_uint4(o[4], o[5], o[6], o[7]);
      }
      act[q] = lo;
      act[kFPlane + q] = hi;
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    // conv3's 1x1 MMA: Z[q][tap] for every block
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int b = 0; b < kFBlocks; ++b) cnn_mma(tmem + 16 * b, da + (kFQ2 + 128 * b), db3, 0u);
      cnn_commit(bar);
    }
    got = warp == 0 ? mbar_wait(bar, phase) : true;
    if (__syncthreads_or(!got)) {
      ok = false;
      break;
    }
    phase ^= 1u;
    tc_fence_after();
    // partials into the activation buffer (h2 is consumed): z_s[tap][q - kFQ2]
    float* zs = reinterpret_cast<float*>(smf + kFSmAct);
    for (int b = warp >> 2; b < kFBlocks; b += kFGroups) {
      float v[16];
      cnn_tmem_ld16(tmem + ((uint32_t)(32 * lq) << 16) + 16 * b, v);
      const int qi = 128 * b + 32 * lq + lane;
#pragma unroll
      for (int t = 0; t < 9; ++t) zs[t * kFZ + qi] = v[t];
    }
    tc_fence_before();
    __syncthreads();
    // y = x + (b3 + sum_tap Z[p + (dy, dx)][tap])
    float* ym = y + (size_t)im * h * w;
    const float sc = scale ? __ldg(&scale[im]) : 1.f;
    for (int k = tid; k < kFTh * kFTw; k += kFThreads) {
      const int ry = k / kFTw, rx = k - ry * kFTw;
      const int iy = y0 + ry, ix = x0 + rx;
      if (iy >= h || ix >= w) continue;
      const int q = (ry + 3) * kFWt + rx + 3;
      float z = b3;
#pragma unroll
      for (int t = 0; t < 9; ++t) z += zs[t * kFZ + q + tap_dy(t) * kFWt + tap_dx(t) - kFQ2];
      ym[(size_t)iy * w + ix] = (xs[q] + z) * sc;
    }
    __syncthreads();  // x and the partials are read before the next tile overwrites them
  }
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
    // the MMAs in flight finish before the tensor memory is released
    if (warp == 0) mbar_wait(bar, phase);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "n"(kFTmemCols)
                 : "memory");
}

int cnn_check(int n_img, int h, int w) {
  if (n_img < 1 || h < 1 || w < 1 || n_img > 65535 || h > 65535)
    return fail(GR_ERR_ARG, "cnn: need 1 <= n_img, h <= 65535 and w >= 1");
  return GR_OK;
}

}  // namespace
}  // namespace gr

using namespace gr;

extern "C" {

int gr_cnn_param_count(void) { return kCnnParams; }

size_t gr_cnn_workspace_bytes(int n_img, int h, int w) {
  if (n_img < 1 || h < 1 || w < 1) return 0;
  const size_t px = (size_t)n_img * h * w;
  // h1, h2, gz1, gz2 (bf16 x 16) + gy (f32) + block partials + loss partials
  return 4 * px * kC * 2 + px * 4 + wg_blocks_bound(n_img, h, w) * kCnnParams * 4 + 1024 * 8 + 1024;
}

size_t gr_cnn_forward_workspace_bytes(int n_img, int h, int w) {
  return 2 * (size_t)n_img * h * w * kC * 2;  // h1, h2 (BF16 x 16)
}

int gr_cnn_forward(const float* params, const float* x, float* y, int n_img, int h, int w,
                   void* workspace, void* stream) {
  int rc = cnn_check(n_img, h, w);
  if (rc) return rc;
  if (!params || !x || !y || !workspace) return fail(GR_ERR_ARG, "cnn forward: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t px = (size_t)n_img * h * w;
  __nv_bfloat16* h1 = static_cast<__nv_bfloat16*>(workspace);
  __nv_bfloat16* h2 = h1 + px * kC;
  const dim3 gp((w + 127) / 128, (h + kThinPx - 1) / kThinPx, n_img);
  cnn_conv1_kernel<<<gp, 128, 0, st>>>(params, x, h1, h, w);
  const int s2 = strip_segments(n_img, h, w, kStBlocks);
  const dim3 g2((w + kStW - 1) / kStW * s2, n_img);
  cnn_conv2_kernel<<<g2, kStThreads, 0, st>>>(params, h1, nullptr, h2, h, w, 0, s2);
  cnn_conv3_kernel<<<dim3((w + 128 * kThinPx - 1) / (128 * kThinPx), (h + kConv3Rows - 1) / kConv3Rows, n_img), 128, 0, st>>>(
      params, x, h2, y, h, w);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "cnn forward: %s", cudaGetErrorString(e));
}

int gr_cnn_backward(const float* params, const float* x, const float* y, const float* target,
                    int n_img, int h, int w, float* grads, double* loss, void* workspace,
                    void* stream) {
  int rc = cnn_check(n_img, h, w);
  if (rc) return rc;
  if (!params || !x || !y || !target || !grads || !workspace)
    return fail(GR_ERR_ARG, "cnn backward: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t px = (size_t)n_img * h * w;
  __nv_bfloat16* h1 = static_cast<__nv_bfloat16*>(workspace);
  __nv_bfloat16* h2 = h1 + px * kC;
  __nv_bfloat16* gz1 = h2 + px * kC;
  __nv_bfloat16* gz2 = gz1 + px * kC;
  float* gy = reinterpret_cast<float*>(gz2 + px * kC);
  const int segs = wg_segments(n_img, h, w);
  const long blocks = wg_blocks(n_img, h, w);
  float* part = gy + px;
  double* lpart = reinterpret_cast<double*>(part + (size_t)blocks * kCnnParams);
  lpart = reinterpret_cast<double*>(((uintptr_t)lpart + 7) & ~(uintptr_t)7);
  const int lblocks = 1024;
  cnn_loss_kernel<<<lblocks, 256, 0, st>>>(y, target, gy, lpart, (long)px);
  const dim3 gp((w + 127) / 128, (h + kThinPx - 1) / kThinPx, n_img);
  cnn_conv3_bwd_kernel<<<gp, 128, 0, st>>>(params, gy, h2, gz2, h, w);
  const int s2 = strip_segments(n_img, h, w, kStBlocks);
  cnn_conv2_kernel<<<dim3((w + kStW - 1) / kStW * s2, n_img), kStThreads, 0, st>>>(params, gz2, h1, gz1,
                                                                                  h, w, 1, s2);
  cudaError_t e = cudaFuncSetAttribute(cnn_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(WgSmem));
  if (e != cudaSuccess) return fail(GR_ERR_CUDA, "cnn backward: %s", cudaGetErrorString(e));
  cnn_wgrad_kernel<<<dim3((unsigned)(blocks / n_img), n_img), kWgThreads, sizeof(WgSmem), st>>>(
      x, gy, h1, h2, gz1, gz2, part, h, w, segs);
  cnn_reduce_kernel<<<(kCnnParams + 31) / 32, 256, 0, st>>>(part, blocks, grads);
  if (loss) {
    double lp[lblocks];
    e = cudaMemcpyAsync(lp, lpart, sizeof(lp), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(GR_ERR_CUDA, "cnn loss: %s", cudaGetErrorString(e));
    double s = 0.0;
    for (int i = 0; i < lblocks; ++i) s += lp[i];
    *loss = s / (double)px;
  }
  e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "cnn backward: %s", cudaGetErrorString(e));
}

size_t gr_cnn_infer_workspace_bytes(void) { return 256; }

int gr_cnn_infer(const float* params, const float* x, float* y, const float* scale, int n_img,
                 int h, int w, void* workspace, void* stream) {
  int rc = cnn_check(n_img, h, w);
  if (rc) return rc;
  if (!params || !x || !y || !workspace) return fail(GR_ERR_ARG, "cnn infer: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(cnn_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kFSmemLaunch);
  if (e != cudaSuccess) return fail(GR_ERR_CUDA, "cnn infer: %s", cudaGetErrorString(e));
  const long tiles = (long)n_img * ((h + kFTh - 1) / kFTh) * ((w + kFTw - 1) / kFTw);
  const int blocks = (int)std::min<long>(tiles, (long)kFCtas * sms);
  cnn_fused_kernel<<<blocks, kFThreads, kFSmemLaunch, st>>>(params, x, y, scale, n_img, h, w,
                                                            static_cast<int*>(workspace));
  e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "cnn infer: %s", cudaGetErrorString(e));
}

int gr_cnn_infer_status(void* workspace, void* stream) {
  if (!workspace) return fail(GR_ERR_ARG, "cnn infer status: null workspace");
  cudaStream_t st = (cudaStream_t)stream;
  int flag = 0;
  cudaError_t e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaMemcpy(&flag, workspace, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && flag) e = cudaMemset(workspace, 0, sizeof(int));
  if (e != cudaSuccess) return fail(GR_ERR_CUDA, "cnn infer status: %s", cudaGetErrorString(e));
  return flag ? fail(GR_ERR_TIMEOUT, "cnn infer: a bounded device wait ran out") : GR_OK;
}

int gr_cnn_adam(float* params, const float* grads, float* m, float* v, int step, float lr,
                float beta1, float beta2, float eps, void* stream) {
  if (!params || !grads || !m || !v || step < 1) return fail(GR_ERR_ARG, "cnn adam: bad arguments");
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  cnn_adam_kernel<<<(kCnnParams + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
      params, grads, m, v, kCnnParams, lr, beta1, beta2, eps, c1, c2);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GR_OK : fail(GR_ERR_CUDA, "cnn adam: %s", cudaGetErrorString(e));
}

}  // extern "C"
