// Fused softmax cross-entropy over large vocabularies: logits[rows, V] (bf16 or fp32) and integer
// labels -> per-row loss and log-sum-exp (forward); dlogits = (softmax - onehot) * dloss (backward).
// Replaces log_softmax + nll_loss (keras/src/backend/torch/nn.py:936-982) and their fp32 upcast copies.
#define XE_EXP __expf
#include "xent_rows.cuh"

constexpr int XE_THREADS = 512;

// `ld` is the row pitch in elements (>= V).  When rows start 16-byte aligned (`vec` = 1: base pointer aligned and the pitch a
// multiple of 16 bytes) the body is read and written as 16-byte vectors; the tail and unaligned inputs use scalar accesses.
// Backward also zeroes the columns [V, Vz) of each row: a padded logits buffer gets a gradient that a padded GEMM can consume.
template <typename T>
__global__ void __launch_bounds__(XE_THREADS) xent_fwd_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                              float* __restrict__ loss, float* __restrict__ lse_out, int V, long long ld, int vec) {
  __shared__ float red[32];
  constexpr int VN = XeVec<T>::N;
  const long long row = blockIdx.x;
  const T* l = logits + row * ld;
  float m = XE_LOWEST, s = 0.f;
  const int body = vec ? (V / VN) * VN : 0;
  for (int i = threadIdx.x * VN; i < body; i += XE_THREADS * VN) {
    float v[VN];
    xe_load<T>(l + i, v);
    float vm = v[0];
#pragma unroll
    for (int j = 1; j < VN; ++j) vm = fmaxf(vm, v[j]);
    if (vm > m) {
      s *= __expf(m - vm);
      m = vm;
    }
#pragma unroll
    for (int j = 0; j < VN; ++j) s += __expf(v[j] - m);
  }
  for (int i = body + threadIdx.x; i < V; i += XE_THREADS) xe_online(to_f32<T>(l[i]), m, s);
  const float gm = block_max(m, red);
  s *= __expf(m - gm);
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    const float lse = gm + logf(s);
    const long long t = labels[row];
    lse_out[row] = lse;
    loss[row] = (t >= 0 && t < V) ? lse - to_f32<T>(l[t]) : 0.f;
  }
}

// One row's gradient by the threads of a block.
template <typename T>
__device__ __forceinline__ void xe_row_gradient(const T* __restrict__ l, T* __restrict__ d, float r_lse, long long t, float g, int V, int Vz, int vec) {
  constexpr int VN = XeVec<T>::N;
  const int body = vec ? (V / VN) * VN : 0;
  for (int i = threadIdx.x * VN; i < body; i += XE_THREADS * VN) {
    float v[VN];
    xe_load<T>(l + i, v);
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      float p = __expf(v[j] - r_lse);
      if (i + j == t) p -= 1.f;
      v[j] = p * g;
    }
    xe_store<T>(d + i, v);
  }
  for (int i = body + threadIdx.x; i < Vz; i += XE_THREADS) {
    float p = 0.f;
    if (i < V) {
      p = __expf(to_f32<T>(l[i]) - r_lse);
      if (i == t) p -= 1.f;
    }
    d[i] = from_f32<T>(p * g);
  }
}

// Loss and gradient of a row in one visit, for a caller that knows which upstream gradient `g` is coming (the mean over the rows): the second
// reading of the row, 100 KB at a vocabulary of 50257, is served by L2, so the logits cross the memory bus once and not twice.  The
// backward kernel still looks at the gradient that really comes, row by row, and computes the rows that it differs in.
// [16384, 50257] bf16: forward and backward 293 + 524 -> 684 + 4 us; 3.3 GB take 504.
template <typename T>
__global__ void __launch_bounds__(XE_THREADS) xent_fwd_grad_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                                   float* __restrict__ loss, float* __restrict__ lse_out, T* __restrict__ dlogits, float g0, int V,
                                                                   long long ld, int Vz, int vec) {
  __shared__ float red[32];
  constexpr int VN = XeVec<T>::N;
  const long long row = blockIdx.x;
  const T* l = logits + row * ld;
  T* d = dlogits + row * ld;
  const long long t = labels[row];
  const bool valid = t >= 0 && t < V;
  const float g = valid ? g0 : 0.f;
  float m = XE_LOWEST, s = 0.f;
  const int body = vec ? (V / VN) * VN : 0;
  for (int i = threadIdx.x * VN; i < body; i += XE_THREADS * VN) {
    float v[VN];
    xe_load<T>(l + i, v);
    float vm = v[0];
#pragma unroll
    for (int j = 1; j < VN; ++j) vm = fmaxf(vm, v[j]);
    if (vm > m) {
      s *= __expf(m - vm);
      m = vm;
    }
#pragma unroll
    for (int j = 0; j < VN; ++j) s += __expf(v[j] - m);
  }
  for (int i = body + threadIdx.x; i < V; i += XE_THREADS) xe_online(to_f32<T>(l[i]), m, s);
  const float gm = block_max(m, red);
  s *= __expf(m - gm);
  s = block_sum(s, red);
  const float lse = gm + logf(s);
  if (threadIdx.x == 0) {
    lse_out[row] = lse;
    loss[row] = valid ? lse - to_f32<T>(l[t]) : 0.f;
  }
  xe_row_gradient<T>(l, d, lse, t, g, V, Vz, vec);
}

template <typename T>
__global__ void __launch_bounds__(XE_THREADS) xent_bwd_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                              const float* __restrict__ lse, const float* __restrict__ dloss, int ds, T* __restrict__ dlogits,
                                                              int V, long long ld, int Vz, int vec) {
  const long long row = blockIdx.x;
  const long long t = labels[row];
  xe_row_gradient<T>(logits + row * ld, dlogits + row * ld, lse[row], t, t >= 0 && t < V ? dloss[row * ds] : 0.f, V, Vz, vec);
}

// The rows hold the gradient for an upstream gradient of g0: those that another one reaches are computed again.  XE_CHECKED rows a block,
// looked at by a thread each: [16384, 50257] 4 us where nothing differs.
constexpr int XE_CHECKED = 64;
template <typename T>
__global__ void __launch_bounds__(XE_THREADS) xent_bwd_check_kernel(const T* __restrict__ logits, const long long* __restrict__ labels,
                                                                    const float* __restrict__ lse, const float* __restrict__ dloss, int ds, T* __restrict__ dlogits,
                                                                    long long rows, int V, long long ld, int Vz, int vec, float g0) {
  __shared__ unsigned char again[XE_CHECKED];
  const long long first = (long long)blockIdx.x * XE_CHECKED;
  int any = 0;
  if (threadIdx.x < XE_CHECKED) {
    const long long row = first + threadIdx.x;
    if (row < rows) {
      const long long t = labels[row];
      any = t >= 0 && t < V && dloss[row * ds] != g0;  // a NaN differs
    }
    again[threadIdx.x] = (unsigned char)any;
  }
  if (!__syncthreads_or(any)) return;
  for (int i = 0; i < XE_CHECKED; ++i) {
    if (!again[i]) continue;
    const long long row = first + i;
    xe_row_gradient<T>(logits + row * ld, dlogits + row * ld, lse[row], labels[row], dloss[row * ds], V, Vz, vec);
  }
}

// xent_classes.cu
constexpr int XE_FEW = 64;
int kb200_xent_classes_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, long long ld, int vec, int dtype,
                           int* outside, cudaStream_t stream);
int kb200_xent_classes_bwd(const void* logits, const long long* labels, const float* lse, const float* dloss, int dloss_stride, void* dlogits, long long rows, int V,
                           long long ld, int zero_to, int vec, int dtype, cudaStream_t stream);

// outside: an int in host memory that the kernel can write, set where fewer than 64 classes meet a label that is none of them (nor the ignored
// -100); or null.
KB_API int kb200_xent_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, long long ld, int dtype, int* outside,
                          cudaStream_t stream) {
  if (rows <= 0) return 0;
  const int esize = dtype == 1 ? 2 : 4;
  const int vec = (((uintptr_t)logits & 15) == 0 && (ld * esize) % 16 == 0) ? 1 : 0;
  if (V < XE_FEW && rows * 32 < (1ll << 38)) return kb200_xent_classes_fwd(logits, labels, loss, lse, rows, V, ld, vec, dtype, outside, stream);
  if (V <= XE_NARROW && rows * 32 < (1ll << 38)) {
    if (dtype == 1) xe_narrow_fwd<__nv_bfloat16>((const __nv_bfloat16*)logits, labels, loss, lse, rows, V, ld, vec, stream);
    else xe_narrow_fwd<float>((const float*)logits, labels, loss, lse, rows, V, ld, vec, stream);
  } else if (dtype == 1)
    xent_fwd_kernel<__nv_bfloat16><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, labels, loss, lse, V, ld, vec);
  else
    xent_fwd_kernel<float><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const float*)logits, labels, loss, lse, V, ld, vec);
  KB_CHECK_LAUNCH("xent_fwd");
  return 0;
}

// Rows wide enough for kb200_xent_fwd_grad: narrower ones have little to gain.
KB_API int kb200_xent_wide(int V) { return V > XE_NARROW ? 1 : 0; }

// As kb200_xent_fwd, and dlogits for an upstream gradient of g0 in every row; kb200_xent_bwd with done = 1 and the same g0 completes it.
KB_API int kb200_xent_fwd_grad(const void* logits, const long long* labels, float* loss, float* lse, void* dlogits, float g0, long long rows, int V, long long ld,
                               int zero_to, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  const int esize = dtype == 1 ? 2 : 4;
  const int vec = ((((uintptr_t)logits | (uintptr_t)dlogits) & 15) == 0 && (ld * esize) % 16 == 0) ? 1 : 0;
  if (zero_to < V) zero_to = V;
  if (dtype == 1)
    xent_fwd_grad_kernel<__nv_bfloat16><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, labels, loss, lse, (__nv_bfloat16*)dlogits, g0, V, ld,
                                                                                     zero_to, vec);
  else
    xent_fwd_grad_kernel<float><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const float*)logits, labels, loss, lse, (float*)dlogits, g0, V, ld, zero_to, vec);
  KB_CHECK_LAUNCH("xent_fwd_grad");
  return 0;
}

// `zero_to` (V <= zero_to <= ld): columns [V, zero_to) of every dlogits row are written as zeros.  done: dlogits come from
// kb200_xent_fwd_grad with this g0.  dloss_stride: 1, or 0 where every row has the one upstream gradient.
KB_API int kb200_xent_bwd(const void* logits, const long long* labels, const float* lse, const float* dloss, int dloss_stride, void* dlogits, long long rows, int V,
                          long long ld, int zero_to, int done, float g0, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  const int esize = dtype == 1 ? 2 : 4;
  const int vec = ((((uintptr_t)logits | (uintptr_t)dlogits) & 15) == 0 && (ld * esize) % 16 == 0) ? 1 : 0;
  if (zero_to < V) zero_to = V;
  if (V < XE_FEW && !done && rows * 32 < (1ll << 38))
    return kb200_xent_classes_bwd(logits, labels, lse, dloss, dloss_stride, dlogits, rows, V, ld, zero_to, vec, dtype, stream);
  if (done) {
    const unsigned grid = (unsigned)((rows + XE_CHECKED - 1) / XE_CHECKED);
    if (dtype == 1)
      xent_bwd_check_kernel<__nv_bfloat16><<<grid, XE_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, labels, lse, dloss, dloss_stride, (__nv_bfloat16*)dlogits, rows, V, ld,
                                                                              zero_to, vec, g0);
    else
      xent_bwd_check_kernel<float><<<grid, XE_THREADS, 0, stream>>>((const float*)logits, labels, lse, dloss, dloss_stride, (float*)dlogits, rows, V, ld, zero_to, vec, g0);
  } else if (V <= XE_NARROW && rows * 32 < (1ll << 38)) {
    if (dtype == 1)
      xe_narrow_bwd<__nv_bfloat16>((const __nv_bfloat16*)logits, labels, lse, dloss, dloss_stride, (__nv_bfloat16*)dlogits, rows, V, ld, zero_to, vec, stream);
    else
      xe_narrow_bwd<float>((const float*)logits, labels, lse, dloss, dloss_stride, (float*)dlogits, rows, V, ld, zero_to, vec, stream);
  } else if (dtype == 1)
    xent_bwd_kernel<__nv_bfloat16><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, labels, lse, dloss, dloss_stride, (__nv_bfloat16*)dlogits, V,
                                                                                ld, zero_to, vec);
  else
    xent_bwd_kernel<float><<<(unsigned)rows, XE_THREADS, 0, stream>>>((const float*)logits, labels, lse, dloss, dloss_stride, (float*)dlogits, V, ld, zero_to, vec);
  KB_CHECK_LAUNCH("xent_bwd");
  return 0;
}
