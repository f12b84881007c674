// Row kernels and helpers of the softmax cross-entropy.  Included by xent.cu (vocabularies: XE_EXP is the fast exponential, its error far below
// bf16's rounding and the sum's) and by xent_classes.cu (a handful of classes in full accuracy).
#pragma once
#include "common.cuh"

namespace {
template <typename T>
struct XeVec {
  static constexpr int N = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ void xe_load(const T* p, float* v) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  if constexpr (sizeof(T) == 2) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
  } else {
    const float* f = reinterpret_cast<const float*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = f[j];
  }
}

template <typename T>
__device__ __forceinline__ void xe_store(T* p, const float* v) {
  uint4 raw;
  if constexpr (sizeof(T) == 2) {
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
  } else {
    float* f = reinterpret_cast<float*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) f[j] = v[j];
  }
  *reinterpret_cast<uint4*>(p) = raw;
}

// The running maximum starts at the lowest finite value, not at -inf: a masked class (-inf) then adds exp(-inf) = 0 from the first on, and
// needs no test of its own (one in this loop cost [16384, 50257] fp32 520 -> 1176 us).
constexpr float XE_LOWEST = -3.402823466e38f;

// Labels outside the classes.  A vocabulary's are ignored: loss and gradient zero.  A classifier's (`strict`) are mistakes, but for the -100 that the
// library's loss ignores: both are NaN, and the host is told through `outside` (in its memory; may be null).
constexpr long long XE_IGNORED = -100;
__device__ __forceinline__ bool xe_mistaken(long long t, int V, int strict) { return strict && (t < 0 || t >= V) && t != XE_IGNORED; }
__device__ __forceinline__ void xe_online(float v, float& m, float& s) {
  if (v > m) {
    s = s * XE_EXP(m - v) + 1.f;
    m = v;
  } else {
    s += XE_EXP(v - m);
  }
}

// Narrow rows (at most XE_NARROW columns: classifiers, per-pixel labels).  A CTA per row leaves most of its 512 threads without a
// column and pays two block-wide reductions for a row of a few hundred bytes; here G lanes of a warp share a row, so a warp
// holds 32 / G rows and the reductions are shuffles.  Bound by the logits' traffic.  [200704, 64] bf16 (25.7 MB of logits):
// forward 569 -> 9 us, backward 321 -> 13 us.
constexpr int XE_NARROW = 2048;  // 8 vectors a lane at G = 32; beyond it a CTA per row has work for all of its warps

template <typename T, int G>
__global__ void __launch_bounds__(256) xent_narrow_fwd_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                              float* __restrict__ loss, float* __restrict__ lse_out, long long rows, int V, long long ld,
                                                              int vec, int strict, int* outside) {
  constexpr int VN = XeVec<T>::N;
  const int gl = threadIdx.x & (G - 1);
  const long long row = (long long)blockIdx.x * (256 / G) + threadIdx.x / G;
  const bool live = row < rows;  // no early exit: every lane takes part in the shuffles
  const T* l = logits + (live ? row : 0) * ld;
  const int n = live ? V : 0;
  const int body = vec ? (n / VN) * VN : 0;
  float m = XE_LOWEST, s = 0.f;
  for (int i = gl * VN; i < body; i += G * VN) {
    float v[VN];
    xe_load<T>(l + i, v);
    float vm = v[0];
#pragma unroll
    for (int j = 1; j < VN; ++j) vm = fmaxf(vm, v[j]);
    if (vm > m) {
      s *= XE_EXP(m - vm);
      m = vm;
    }
#pragma unroll
    for (int j = 0; j < VN; ++j) s += XE_EXP(v[j] - m);
  }
  for (int i = body + gl; i < n; i += G) xe_online(to_f32<T>(l[i]), m, s);
  float gm = m;
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
  s *= XE_EXP(m - gm);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (live && gl == 0) {
    const float lse = gm + logf(s);
    const long long t = labels[row];
    const bool mistaken = xe_mistaken(t, V, strict);
    lse_out[row] = lse;
    loss[row] = (t >= 0 && t < V) ? lse - to_f32<T>(l[t]) : mistaken ? NAN : 0.f;
    if (mistaken && outside != nullptr) *reinterpret_cast<volatile int*>(outside) = 1;
  }
}

template <typename T, int G>
__global__ void __launch_bounds__(256) xent_narrow_bwd_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                              const float* __restrict__ lse, const float* __restrict__ dloss, int ds, T* __restrict__ dlogits,
                                                              long long rows, int V, long long ld, int Vz, int vec, int strict) {
  constexpr int VN = XeVec<T>::N;
  const int gl = threadIdx.x & (G - 1);
  const long long row = (long long)blockIdx.x * (256 / G) + threadIdx.x / G;
  if (row >= rows) return;
  const T* l = logits + row * ld;
  T* d = dlogits + row * ld;
  const float r_lse = lse[row];
  const long long t = labels[row];
  const float g = (t >= 0 && t < V) ? dloss[row * ds] : xe_mistaken(t, V, strict) ? NAN : 0.f;
  const int body = vec ? (V / VN) * VN : 0;
  for (int i = gl * VN; i < body; i += G * VN) {
    float v[VN];
    xe_load<T>(l + i, v);
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      float p = XE_EXP(v[j] - r_lse);
      if (i + j == t) p -= 1.f;
      v[j] = p * g;
    }
    xe_store<T>(d + i, v);
  }
  for (int i = body + gl; i < Vz; i += G) {
    float p = 0.f;
    if (i < V) {
      p = XE_EXP(to_f32<T>(l[i]) - r_lse);
      if (i == t) p -= 1.f;
    }
    d[i] = from_f32<T>(p * g);
  }
}

// Lanes a row: enough that each has one vector (or, on the scalar path, a handful of elements), never more than a warp.
static int xe_lanes(int V, int vec, int vn) {
  const int items = vec ? (V + vn - 1) / vn : (V + 3) / 4;
  return items <= 4 ? 4 : items <= 8 ? 8 : items <= 16 ? 16 : 32;
}

template <typename T>
static void xe_narrow_fwd(const T* logits, const long long* labels, float* loss, float* lse, long long rows, int V, long long ld, int vec, cudaStream_t st,
                          int strict = 0, int* outside = nullptr) {
  const int g = xe_lanes(V, vec, XeVec<T>::N);
  const unsigned grid = (unsigned)((rows * g + 255) / 256);
  if (g == 4) xent_narrow_fwd_kernel<T, 4><<<grid, 256, 0, st>>>(logits, labels, loss, lse, rows, V, ld, vec, strict, outside);
  else if (g == 8) xent_narrow_fwd_kernel<T, 8><<<grid, 256, 0, st>>>(logits, labels, loss, lse, rows, V, ld, vec, strict, outside);
  else if (g == 16) xent_narrow_fwd_kernel<T, 16><<<grid, 256, 0, st>>>(logits, labels, loss, lse, rows, V, ld, vec, strict, outside);
  else xent_narrow_fwd_kernel<T, 32><<<grid, 256, 0, st>>>(logits, labels, loss, lse, rows, V, ld, vec, strict, outside);
}

template <typename T>
static void xe_narrow_bwd(const T* logits, const long long* labels, const float* lse, const float* dloss, int ds, T* dlogits, long long rows, int V, long long ld,
                          int Vz, int vec, cudaStream_t st, int strict = 0) {
  const int g = xe_lanes(V, vec, XeVec<T>::N);
  const unsigned grid = (unsigned)((rows * g + 255) / 256);
  if (g == 4) xent_narrow_bwd_kernel<T, 4><<<grid, 256, 0, st>>>(logits, labels, lse, dloss, ds, dlogits, rows, V, ld, Vz, vec, strict);
  else if (g == 8) xent_narrow_bwd_kernel<T, 8><<<grid, 256, 0, st>>>(logits, labels, lse, dloss, ds, dlogits, rows, V, ld, Vz, vec, strict);
  else if (g == 16) xent_narrow_bwd_kernel<T, 16><<<grid, 256, 0, st>>>(logits, labels, lse, dloss, ds, dlogits, rows, V, ld, Vz, vec, strict);
  else xent_narrow_bwd_kernel<T, 32><<<grid, 256, 0, st>>>(logits, labels, lse, dloss, ds, dlogits, rows, V, ld, Vz, vec, strict);
}
}  // namespace
