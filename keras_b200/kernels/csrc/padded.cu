// Matrices whose width is no multiple of 8 (a 50257-word vocabulary) against the GEMM's rows of 16-byte pitch: zero-padding a bf16
// matrix, and adding a padded bf16 gradient to the fp32 matrix it belongs to; and the copy of a batch with its rounding.  Both are bound by their traffic; the library's kernels
// for them fall back to scalar indexing because one side's rows start at odd addresses.
// [768, 50257]: pad 109 (fill and copy) -> 33 us, add 148 -> 65 us; the traffic takes 23 and 58 us.
#include "common.cuh"

namespace {
constexpr int THREADS = 256;

// dst [rows, wide] = src [rows, cols] with zeros behind; one 16-byte store a thread
__global__ void __launch_bounds__(THREADS) pad_columns_kernel(const unsigned short* __restrict__ src, uint4* __restrict__ dst, int rows, int cols, int vecs) {
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const unsigned short* s = src + (size_t)r * cols;
    for (int v = blockIdx.x * THREADS + threadIdx.x; v < vecs; v += gridDim.x * THREADS) {
      unsigned e[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = v * 8 + k < cols ? s[v * 8 + k] : 0;
      dst[(size_t)r * vecs + v] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
    }
  }
}

// dst [rows, cols] += src [rows, cols] of row pitch ld; neighbouring lanes take neighbouring columns, four rows of loads in flight
__global__ void __launch_bounds__(THREADS) add_rows_kernel(const __nv_bfloat16* __restrict__ src, long long ld, float* __restrict__ dst, int rows, int cols) {
  constexpr int U = 4;
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const __nv_bfloat16* s = src + r * ld;
    float* d = dst + (size_t)r * cols;
    for (int c0 = blockIdx.x * THREADS * U + threadIdx.x; c0 < cols; c0 += gridDim.x * THREADS * U) {
      float a[U], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + u * THREADS;
        a[u] = c < cols ? __bfloat162float(s[c]) : 0.f;
        b[u] = c < cols ? d[c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c0 + u * THREADS < cols) d[c0 + u * THREADS] = a[u] + b[u];
    }
  }
}

// A batch on its way into a recorded step: its copy and its bf16 rounding from one read.  [256, 56, 56, 256]: copy 251 us and cast 174 us
// -> 349 us together; the 2.06 GB take 310.  Where the step reads nothing but the rounding, the copy is left out (dst null): 180 us, 1.23 GB.
__global__ void __launch_bounds__(THREADS) copy_cast_kernel(const float4* __restrict__ src, float4* __restrict__ dst, uint4* __restrict__ dst16, long long vecs) {
  constexpr int U = 2;
  const long long step = (long long)gridDim.x * THREADS;
  for (long long v0 = (long long)blockIdx.x * THREADS + threadIdx.x; v0 < vecs; v0 += step * U) {
    float4 a[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v0 + u * step < vecs) a[u][0] = src[2 * (v0 + u * step)], a[u][1] = src[2 * (v0 + u * step) + 1];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long v = v0 + u * step;
      if (v < vecs) {
        if (dst != nullptr) dst[2 * v] = a[u][0], dst[2 * v + 1] = a[u][1];
        const float f[8] = {a[u][0].x, a[u][0].y, a[u][0].z, a[u][0].w, a[u][1].x, a[u][1].y, a[u][1].z, a[u][1].w};
        const bf16x8 h = pack8(f);
        dst16[v] = reinterpret_cast<const uint4&>(h);
      }
    }
  }
}

dim3 row_grid(int rows, int per_row) {
  const int blocks = (per_row + THREADS - 1) / THREADS;
  return dim3((unsigned)(blocks < 1 ? 1 : blocks > 65535 ? 65535 : blocks), (unsigned)(rows < 65535 ? rows : 65535));
}
}  // namespace

// src: bf16 [rows, cols] contiguous; dst: bf16 [rows, wide], wide a multiple of 8, 16-byte aligned
KB_API int kb200_pad_columns(const void* src, void* dst, int rows, int cols, int wide, cudaStream_t stream) {
  if (rows <= 0 || wide <= 0) return 0;
  if (wide % 8 || cols > wide || ((uintptr_t)dst & 15)) {
    kb200_set_error("pad_columns: the result's rows must be multiples of 16 bytes and hold the source's");
    return -2;
  }
  pad_columns_kernel<<<row_grid(rows, wide / 8), THREADS, 0, stream>>>((const unsigned short*)src, (uint4*)dst, rows, cols, wide / 8);
  KB_CHECK_LAUNCH("pad_columns");
  return 0;
}

// dst: fp32 [rows, cols] contiguous += src: bf16 [rows, cols] of row pitch ld
KB_API int kb200_add_rows(const void* src, long long ld, float* dst, int rows, int cols, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  add_rows_kernel<<<row_grid(rows, (cols + 3) / 4), THREADS, 0, stream>>>((const __nv_bfloat16*)src, ld, dst, rows, cols);
  KB_CHECK_LAUNCH("add_rows");
  return 0;
}

// dst = src (unless null) and dst16 = its rounding to bf16: n values, a multiple of 8, all 16-byte aligned
KB_API int kb200_copy_cast(const void* src, void* dst, void* dst16, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 || (((uintptr_t)src | (uintptr_t)dst | (uintptr_t)dst16) & 15)) {
    kb200_set_error("copy_cast: values in multiples of 8, 16-byte aligned");
    return -2;
  }
  const long long blocks = (n / 8 + THREADS - 1) / THREADS, most = (long long)kb_sm_count() * 16;
  copy_cast_kernel<<<(unsigned)(blocks < most ? blocks : most), THREADS, 0, stream>>>((const float4*)src, (float4*)dst, (uint4*)dst16, n / 8);
  KB_CHECK_LAUNCH("copy_cast");
  return 0;
}
