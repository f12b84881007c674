// Shared helpers for the sm_100a kernel library: error reporting, warp/block reductions,
// bf16 vector loads, bounded spin-waits.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define KB_API extern "C" __attribute__((visibility("default")))

// Launch-status convention: every launcher returns 0 on success, else a negative code and sets a
// message retrievable through kb200_last_error().
void kb200_set_error(const char* msg);

#define KB_CHECK_LAUNCH(what)                                   \
  do {                                                          \
    cudaError_t e__ = cudaGetLastError();                       \
    if (e__ != cudaSuccess) {                                   \
      kb200_set_error(cudaGetErrorString(e__));                 \
      return -1;                                                \
    }                                                           \
  } while (0)

// Per-device launcher state.  Kernel attributes and SM counts belong to a device, and one process may drive several:
// every "done once" flag in the launchers is an array indexed by the current device.
constexpr int KB_MAX_DEVICES = 64;

inline int kb_device_slot() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= KB_MAX_DEVICES) dev = 0;
  return dev;
}

inline int kb_sm_count() {
  static int sms[KB_MAX_DEVICES] = {0};
  const int slot = kb_device_slot();
  if (sms[slot] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, slot) != cudaSuccess || v <= 0) v = 148;
    sms[slot] = v;
  }
  return sms[slot];
}

// Raise a kernel's dynamic shared-memory limit once per device.  `flags` is a function-local `static bool [KB_MAX_DEVICES]`.
template <typename Kernel>
inline bool kb_allow_smem(Kernel kernel, int bytes, bool* flags) {
  const int slot = kb_device_slot();
  if (!flags[slot]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    flags[slot] = true;
  }
  return true;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; `red` is shared scratch of >= 32 floats. Result valid in every thread.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float r = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (wid == 0) {
    r = warp_sum(r);
    if (lane == 0) red[0] = r;
  }
  __syncthreads();
  r = red[0];
  return r;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float r = (threadIdx.x < nw) ? red[threadIdx.x] : -INFINITY;
  if (wid == 0) {
    r = warp_max(r);
    if (lane == 0) red[0] = r;
  }
  __syncthreads();
  r = red[0];
  return r;
}

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float* f) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Cumulative distribution function of the normal distribution, Phi(v) = erfc(-v / sqrt(2)) / 2, for the exact GELU and its derivative.
// With a = |v| and t = 1 / (1 + 0.35 a):  Phi(-a) = t * 2^(p(t) - a^2 log2(e) / 2), where p is the polynomial of degree 7 that fits
// log2(Phi(-a) e^(a^2/2) / t) on 0 <= a <= 14 with the least maximum error (a linear program over 6000 Chebyshev points gives its
// coefficients; 6e-7 relative, in float32 9e-7 for a < 1 and 2.5e-6 for a < 6, where the exponent's rounding is most of it).  For results
// that are rounded to bf16; those stored as float32 take erff where it is nearer (gemm_sm100.cuh).  Sixteen instructions, two of them on the special-function pipe; 1 + erf(v / sqrt(2))
// takes twice as many and loses its relative accuracy for negative v.  [16384, 3072, 768] with gelu in the epilogue: 90 us, without 67.
__device__ __forceinline__ float normal_cdf(float v) {
  const float a = fabsf(v), t = __fdividef(1.f, fmaf(0.35f, a, 1.f)), x = a * 0.8493218002880191f;  // x^2 = a^2 log2(e) / 2
  float p = -0.2692641317844391f;
  p = fmaf(p, t, 1.0951932668685913f);
  p = fmaf(p, t, -1.4946914911270142f);
  p = fmaf(p, t, 0.5625093579292297f);
  p = fmaf(p, t, -0.06951091438531876f);
  p = fmaf(p, t, 0.5756505131721497f);
  p = fmaf(p, t, 1.4403815269470215f);
  p = fmaf(p, t, -2.840268850326538f);
  const float lower = t * exp2f(fmaf(-x, x, p));
  return v > 0.f ? 1.f - lower : lower;
}
