// FBP comparator: the reference's OptimizedFBP reconstruction class
// (gridrec/GPU/filteredbackprojection.cpp:190-330, a ReconAlgorithm like GridRec)
// on the device.  Row filter: fbp_filter_kernel (gridrec_kernels.cu).  Here:
// pixel-driven backprojection and the C ABI.
//
// Backprojection of pixel (x, y) of the n x n image (row y), as the reference:
//   x = (col - n/2) / (n/2), y = (row - n/2) / (n/2), r = x cos_a + y sin_a,
//   image += filtered[a][(int)((r + 1) n/2)] for -1 <= r < 1, angles in order,
// in float with the reference's operation order (no contraction), so the sample
// chosen for every (pixel, angle) is the reference's (except an index that
// rounds to n, which is clamped to n - 1 instead of reading outside the row).
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "gr_internal.h"

namespace gr {
namespace {

// A block covers kBpTile x 8 R pixels of S slices: the sample a (pixel, angle) takes
// depends on the geometry only, so one index serves all S slices, whose filtered rows are
// interleaved ([angle][k][slice], one S-float load).  A warp covers 8 x 4 pixels, whose
// samples at one angle span a few consecutive elements whatever the direction, and a
// thread R pixels, eight rows apart: R independent chains per angle.
// Bound by the instruction issue: about 8 instructions per (pixel, angle) for the index
// and one load and S additions for the sums.  The index (int)((r + 1) n/2) comes from an
// addition of 2^23 rounded toward zero (exact for 0 <= t < 2^23) instead of a conversion,
// whose pipe runs at a quarter of the rate.  In blocks that lie well inside the unit
// circle -1 < r < 1 holds for every angle, so they skip the range test and the clamp.
// 2 slices of 2048 x 1500: 2.89 ms with the filter, against 7.70 ms for one slice and one
// pixel per thread with a conversion and a range test per sample.
constexpr int kBpTile = 32, kBpThreads = 256;

template <int S>
struct BpVec;
template <>
struct BpVec<1> {
  using T = float;
  static __device__ __forceinline__ void add(float (&a)[1], float v) { a[0] = __fadd_rn(a[0], v); }
};
template <>
struct BpVec<2> {
  using T = float2;
  static __device__ __forceinline__ void add(float (&a)[2], float2 v) {
    a[0] = __fadd_rn(a[0], v.x);
    a[1] = __fadd_rn(a[1], v.y);
  }
};
template <>
struct BpVec<4> {
  using T = float4;
  static __device__ __forceinline__ void add(float (&a)[4], float4 v) {
    a[0] = __fadd_rn(a[0], v.x);
    a[1] = __fadd_rn(a[1], v.y);
    a[2] = __fadd_rn(a[2], v.z);
    a[3] = __fadd_rn(a[3], v.w);
  }
};

template <int S, int R, bool kInside>
__device__ __forceinline__ void bp_angles(const typename BpVec<S>::T* f, const float2* cs, int n,
                                          int n_ang, float h, float x, const float (&y)[R],
                                          float (&acc)[R][S]) {
  using T = typename BpVec<S>::T;
  // the bits of t + 2^23 are 0x4b000000 + floor(t): the offset goes into the row pointer
  const char* row = reinterpret_cast<const char*>(f) - (size_t)0x4b000000u * sizeof(T);
#pragma unroll 4
  for (int a = 0; a < n_ang; ++a, row += (size_t)n * sizeof(T)) {
    const float2 c = cs[a];  // (cos, sin)
    const float xc = __fmul_rn(x, c.x);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float r = __fadd_rn(xc, __fmul_rn(y[i], c.y));
      const float t = __fmul_rn(__fadd_rn(r, 1.f), h);
      unsigned k = __float_as_uint(__fadd_rz(t, 8388608.f));
      if (!kInside) {
        // r just below 1 can round (r + 1) n/2 up to n; the reference then reads
        // the next row (or past its buffer), here the last sample of the row
        if (!(r >= -1.f && r < 1.f)) continue;
        k = min(k, 0x4b000000u + (unsigned)(n - 1));
      }
      BpVec<S>::add(acc[i], __ldg(reinterpret_cast<const T*>(row + (size_t)k * sizeof(T))));
    }
  }
}

template <int S, int R>
__global__ void __launch_bounds__(kBpThreads) fbp_backproject_kernel(const float* filt,
                                                                     const float2* cs,
                                                                     float* recon, int n,
                                                                     int n_ang, bool finite) {
  extern __shared__ float2 s_cs[];
  for (int i = threadIdx.x; i < n_ang; i += kBpThreads) s_cs[i] = cs[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int xi = blockIdx.x * kBpTile + (warp & 3) * 8 + (lane & 7);
  const int yi = blockIdx.y * (8 * R) + (warp >> 2) * 4 + (lane >> 3);
  const float h = (float)n / 2.0f;
  const float x = __fdiv_rn(__fsub_rn((float)xi, h), h);
  float y[R], acc[R][S];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    y[i] = __fdiv_rn(__fsub_rn((float)(yi + 8 * i), h), h);
#pragma unroll
    for (int s = 0; s < S; ++s) acc[i][s] = 0.f;
  }
  // the block's corner farthest from the centre, in units of the half width; 1e-3 covers
  // the rounding of r and of (cos, sin) many times over
  const float cx = fmaxf(fabsf(blockIdx.x * kBpTile - h), fabsf(blockIdx.x * kBpTile + (kBpTile - 1) - h));
  const float cy = fmaxf(fabsf(blockIdx.y * (8 * R) - h), fabsf(blockIdx.y * (8 * R) + (8 * R - 1) - h));
  const bool inside = finite && cx * cx + cy * cy < (1.f - 1e-3f) * (1.f - 1e-3f) * h * h;
  const typename BpVec<S>::T* f =
      reinterpret_cast<const typename BpVec<S>::T*>(filt) + (size_t)blockIdx.z * n_ang * n;
  if (inside) bp_angles<S, R, true>(f, s_cs, n, n_ang, h, x, y, acc);
  else bp_angles<S, R, false>(f, s_cs, n, n_ang, h, x, y, acc);
  if (xi >= n) return;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (yi + 8 * i >= n) break;
#pragma unroll
    for (int s = 0; s < S; ++s)
      recon[(((size_t)blockIdx.z * S + s) * n + yi + 8 * i) * n + xi] = acc[i][s];
  }
}

template <int S, int R>
cudaError_t launch_backproject_r(const float* filt, const float2* cs, float* recon, int n, int n_ang,
                                 bool finite, int groups, int smem, cudaStream_t st) {
  const dim3 grid((n + kBpTile - 1) / kBpTile, (n + 8 * R - 1) / (8 * R), groups);
  fbp_backproject_kernel<S, R><<<grid, kBpThreads, smem, st>>>(filt, cs, recon, n, n_ang, finite);
  return cudaGetLastError();
}

// Four rows per thread where that leaves four blocks per SM, else one (us for 4 / 1 rows:
// 2 slices of 2048 x 1500 2893 / 3656, of 1024 x 720 468 / 481, of 512 x 360 122 / 81, of
// 256 x 180 70 / 27).
template <int S>
cudaError_t launch_backproject(const float* filt, const float2* cs, float* recon, int n, int n_ang,
                               bool finite, int groups, int smem, cudaStream_t st) {
  const long t = (n + kBpTile - 1) / kBpTile;
  return t * t * groups >= 4 * kSMs
             ? launch_backproject_r<S, 4>(filt, cs, recon, n, n_ang, finite, groups, smem, st)
             : launch_backproject_r<S, 1>(filt, cs, recon, n, n_ang, finite, groups, smem, st);
}

// Lets every form of the backprojection use `smem` bytes of shared memory.
cudaError_t allow_backproject_smem(int smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  const void* forms[] = {(const void*)fbp_backproject_kernel<4, 4>, (const void*)fbp_backproject_kernel<4, 1>,
                         (const void*)fbp_backproject_kernel<2, 4>, (const void*)fbp_backproject_kernel<2, 1>,
                         (const void*)fbp_backproject_kernel<1, 4>, (const void*)fbp_backproject_kernel<1, 1>};
  for (const void* f : forms) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      cudaGetLastError();  // not left behind for the next call's launch check
      return e;
    }
  }
  return cudaSuccess;
}

// Slices backprojected together: 4, then 2, then 1 of what is left of a call's chunk.
int bp_group(int slices) { return slices >= 4 ? 4 : (slices >= 2 ? 2 : 1); }

}  // namespace
}  // namespace gr

struct gr_fbp {
  int device = 0, n = 0, n_ang = 0, max_slices = 1;
  bool finite = true;  // every angle is a number: |r| is bounded by the pixel's radius
  float* d_lut = nullptr;
  float2* d_tw = nullptr;
  float2* d_cs = nullptr;
  float* d_filt = nullptr;
};

using namespace gr;

extern "C" {

int gr_fbp_destroy(gr_fbp* f) {
  if (!f) return GR_OK;
  DeviceGuard g(f->device);
  cudaFree(f->d_lut);
  cudaFree(f->d_tw);
  cudaFree(f->d_cs);
  cudaFree(f->d_filt);
  delete f;
  return GR_OK;
}

int gr_fbp_create(int n_det, int n_ang, const float* theta_deg, int max_slices, int device,
                  gr_fbp** out) {
  if (!out || !theta_deg) return fail(GR_ERR_ARG, "fbp: null argument");
  *out = nullptr;
  if (n_det < 16 || n_det > 8192 || (n_det & (n_det - 1)) || n_ang < 1 || max_slices < 1)
    return fail(GR_ERR_ARG, "fbp: n_det a power of two in [16, 8192], n_ang >= 1, max_slices >= 1");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
    return fail(GR_ERR_ARG, "fbp: device %d not available", device);
  DeviceGuard g(device);
  const int n = n_det;
  // Tables as the reference computes them: the degree list to radians as
  // (theta * PI) / 180 stored in float (PI of gridrec/GPU/fft.h:5), sin/cos of
  // that float; the filter 1 - sqrt(|t|) with t = (k - n/2) / (n/2) in float.
  const double kPiRef = 3.1415926535897932385;
  std::vector<float2> cs(n_ang);
  for (int a = 0; a < n_ang; ++a) {
    const float th = (float)((theta_deg[a] * kPiRef) / 180.0);
    cs[a] = make_float2((float)std::cos((double)th), (float)std::sin((double)th));
  }
  std::vector<float> lut(n);
  for (int k = 0; k < n; ++k) {
    const float t = (float)(k - (float)(n / 2)) / ((float)(n / 2));
    lut[k] = (float)(1 - std::sqrt(std::fabs((double)t)));
  }
  const int nhi = std::max(1, n / 64);
  std::vector<float2> tw(64 + nhi);
  for (int e = 0; e < 64; ++e) {
    const double a = 2.0 * M_PI * e / n;
    tw[e] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  for (int f = 0; f < nhi; ++f) {
    const double a = 2.0 * M_PI * 64.0 * f / n;
    tw[64 + f] = make_float2((float)std::cos(a), (float)std::sin(a));
  }
  gr_fbp* p = new gr_fbp;
  p->device = device;
  p->n = n;
  p->n_ang = n_ang;
  p->max_slices = max_slices;
  for (const float2& c : cs) p->finite = p->finite && std::isfinite(c.x) && std::isfinite(c.y);
  cudaError_t e = cudaMalloc(&p->d_lut, n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_tw, tw.size() * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_cs, n_ang * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&p->d_filt, (size_t)max_slices * n_ang * n * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(p->d_lut, lut.data(), n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(p->d_tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(p->d_cs, cs.data(), n_ang * sizeof(float2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = init_kernel_attributes();
  if (e != cudaSuccess) {
    gr_fbp_destroy(p);
    cudaGetLastError();
    return fail(GR_ERR_NOMEM, "fbp create: %s", cudaGetErrorString(e));
  }
  *out = p;
  return GR_OK;
}

int gr_fbp_reconstruct(gr_fbp* f, const float* sinos, int n_slices, float* recons, void* stream) {
  if (!f || !sinos || !recons || n_slices < 1) return fail(GR_ERR_ARG, "fbp: bad arguments");
  DeviceGuard g(f->device);
  cudaStream_t st = (cudaStream_t)stream;
  const int n = f->n;
  const size_t slice_in = (size_t)f->n_ang * n, slice_out = (size_t)n * n;
  const int smem_bp = f->n_ang * (int)sizeof(float2);
  // too many angles for their table: refused before anything runs
  cudaError_t e = allow_backproject_smem(smem_bp);
  if (e != cudaSuccess)
    return fail(GR_ERR_UNSUPPORTED, "fbp: %d angles: %s", f->n_ang, cudaGetErrorString(e));
  for (int s0 = 0; s0 < n_slices;) {
    // whole groups of one size, as many as the filtered-row buffer holds
    const int S = bp_group(std::min(f->max_slices, n_slices - s0));
    const int groups = std::min(f->max_slices, n_slices - s0) / S;
    FbpFilterArgs fa{sinos + s0 * slice_in, f->d_filt, f->d_lut, f->d_tw, n, f->n_ang, groups * S, S};
    e = launch_fbp_filter(fa, st);
    if (e != cudaSuccess) return fail(GR_ERR_CUDA, "fbp filter: %s", cudaGetErrorString(e));
    float* out = recons + s0 * slice_out;
    e = S == 4 ? launch_backproject<4>(f->d_filt, f->d_cs, out, n, f->n_ang, f->finite, groups, smem_bp, st)
        : S == 2 ? launch_backproject<2>(f->d_filt, f->d_cs, out, n, f->n_ang, f->finite, groups, smem_bp, st)
                 : launch_backproject<1>(f->d_filt, f->d_cs, out, n, f->n_ang, f->finite, groups, smem_bp, st);
    if (e != cudaSuccess) return fail(GR_ERR_CUDA, "fbp backprojection: %s", cudaGetErrorString(e));
    s0 += groups * S;
  }
  return GR_OK;
}

}  // extern "C"
