// LayerNorm / RMSNorm forward and backward over the last axis: rows x D, bf16 or fp32 I/O, fp32 math.
// Replaces F.layer_norm / F.rms_norm plus the two cast kernels around them
// (keras/src/ops/nn.py:3035-3069,3151-3210).
//
// Fast path (rows 16-byte aligned, D a multiple of the 16-byte vector, at most 8 vectors per lane): one warp per row,
// the row lives in registers as raw 16-byte vectors, statistics by warp shuffles only (mean first, then the centred
// second moment), one read and one write of every element.  Backward walks rows with a persistent grid, accumulates
// dgamma/dbeta per lane in registers, reduces them across the block's warps in shared memory and writes one partial
// row per block; a second kernel sums the partial rows (fixed order: deterministic).
// General path: one block per row with scalar accesses.
#include "common.cuh"

constexpr int NORM_THREADS = 256;
constexpr int NW_THREADS = 128;  // fast path: 4 warps = 4 rows per block

template <typename T>
struct NVec {
  static constexpr int N = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ void nv_unpack(const uint4& raw, float* v) {
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
__device__ __forceinline__ uint4 nv_pack(const float* v) {
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
  return raw;
}

// VN consecutive fp32 parameters starting at a 16-byte aligned offset
template <int VN>
__device__ __forceinline__ void load_params(const float* __restrict__ p, int idx, float* out) {
#pragma unroll
  for (int q = 0; q < VN / 4; ++q) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p + idx) + q);
    out[4 * q] = f.x;
    out[4 * q + 1] = f.y;
    out[4 * q + 2] = f.z;
    out[4 * q + 3] = f.w;
  }
}

// A row is shared by WPR warps of an NT-thread block (WPR = 1: one warp per row, no block barrier at all); thread t of
// the row group owns vectors t, t + 32*WPR, ... (VPL of them, `nvec` valid in the row).
template <int NT, int WPR>
__device__ __forceinline__ float row_sum(float v, float* red, int row_in_block, int warp_in_row, int lane, int phase) {
  v = warp_sum(v);
  if constexpr (WPR == 1) {
    return v;
  } else {
    // `red`: [2 phases][rows per block][WPR]; alternating phases make one barrier per reduction enough
    float* slot = red + (phase * (NT / 32 / WPR) + row_in_block) * WPR;
    if (lane == 0) slot[warp_in_row] = v;
    __syncthreads();
    float r = 0.f;
#pragma unroll
    for (int w = 0; w < WPR; ++w) r += slot[w];
    return r;
  }
}

template <typename T, int VPL, int NT, int WPR>
__global__ void __launch_bounds__(NT) norm_fwd_warp_kernel(const T* __restrict__ x, const T* __restrict__ res, T* __restrict__ sum_out,
                                                           const float* __restrict__ gamma, const float* __restrict__ beta,
                                                           T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                                                           long long rows, int D, float eps, int rms, int narrow) {
  constexpr int VN = NVec<T>::N;
  constexpr int RPB = NT / 32 / WPR;  // rows per block
  __shared__ float red[2 * RPB * WPR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row_in_block = warp / WPR, warp_in_row = warp % WPR;
  const int t = warp_in_row * 32 + lane;
  long long row = (long long)blockIdx.x * RPB + row_in_block;
  const bool live = row < rows;
  if (WPR == 1 && !live) return;
  if (!live) row = rows - 1;  // keep the barriers uniform; results of the duplicate are not written
  const int nvec = D / VN;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * D);
  uint4 raw[VPL];
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
    const int i = t + k * 32 * WPR;
    raw[k] = i < nvec ? __ldg(xr + i) : make_uint4(0, 0, 0, 0);
  }
  if (res != nullptr) {  // the row is a residual sum, rounded as the addition alone would leave it
    const uint4* rr = reinterpret_cast<const uint4*>(res + row * D);
    uint4 more[VPL];
#pragma unroll
    for (int k = 0; k < VPL; ++k) more[k] = t + k * 32 * WPR < nvec ? __ldg(rr + t + k * 32 * WPR) : make_uint4(0, 0, 0, 0);
    uint4* so = reinterpret_cast<uint4*>(sum_out + row * D);
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      float v[VN], m[VN];
      nv_unpack<T>(raw[k], v);
      nv_unpack<T>(more[k], m);
#pragma unroll
      for (int j = 0; j < VN; ++j) v[j] += m[j];
      raw[k] = nv_pack<T>(v);
      if (live && t + k * 32 * WPR < nvec) so[t + k * 32 * WPR] = raw[k];
    }
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
    float v[VN];
    nv_unpack<T>(raw[k], v);
#pragma unroll
    for (int j = 0; j < VN; ++j) s += v[j];
  }
  const float mean = rms ? 0.f : row_sum<NT, WPR>(s, red, row_in_block, warp_in_row, lane, 0) / D;
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
    if (t + k * 32 * WPR < nvec) {
      float v[VN];
      nv_unpack<T>(raw[k], v);
#pragma unroll
      for (int j = 0; j < VN; ++j) ss += (v[j] - mean) * (v[j] - mean);
    }
  }
  const float rstd = rsqrtf(row_sum<NT, WPR>(ss, red, row_in_block, warp_in_row, lane, 1) / D + eps);
  if (!live) return;
  if (t == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
  uint4* yr = reinterpret_cast<uint4*>(y + row * D);
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
    const int i = t + k * 32 * WPR;
    if (i < nvec) {
      float v[VN], gv[VN], bv[VN];
      nv_unpack<T>(raw[k], v);
      if (gamma) load_params<VN>(gamma, i * VN, gv);
      if (beta) load_params<VN>(beta, i * VN, bv);
#pragma unroll
      for (int j = 0; j < VN; ++j) {
        float o = (v[j] - mean) * rstd;
        if (gamma) o *= narrow ? to_f32<T>(from_f32<T>(gv[j])) : gv[j];
        if (beta) o += narrow ? to_f32<T>(from_f32<T>(bv[j])) : bv[j];
        v[j] = o;
      }
      yr[i] = nv_pack<T>(v);
    }
  }
}

// Bound by loads in flight: a warp holds a row's two or three tensors and 16 sums a vector of its columns, and the fewer registers that
// takes the more rows an SM has on their way.  MB blocks an SM of 128 threads, and vectors that divide the row (three a lane at 768
// columns).  With the gradient of the sum's other reader added on the way: [16384, 768] bf16 30.5 + 10.7 us apart -> 30.3, [2664, 512]
// 8.2 + 2.0 -> 6.9 (four blocks an SM at three vectors spill, 45.6; the other gradient loaded behind the sums, 36.7).
template <typename T, int VPL, int NT, int WPR, int MB = 1>
__global__ void __launch_bounds__(NT, MB) norm_bwd_warp_kernel(const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ gamma,
                                                           const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ dres,
                                                           T* __restrict__ dx, float* __restrict__ partial_dgamma, float* __restrict__ partial_dbeta,
                                                           long long rows, int D, int rms) {
  constexpr int VN = NVec<T>::N;
  constexpr int RPB = NT / 32 / WPR;
  extern __shared__ float nsm[];  // [RPB][D] staging for the cross-row-group reduction of dgamma, then dbeta
  __shared__ float red[2 * RPB * WPR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row_in_block = warp / WPR, warp_in_row = warp % WPR;
  const int t = warp_in_row * 32 + lane;
  const int nvec = D / VN;
  float dg[VPL * VN], db[VPL * VN];
#pragma unroll
  for (int k = 0; k < VPL; ++k)
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      dg[k * VN + j] = 0.f;
      db[k * VN + j] = 0.f;
    }
  const float inv_d = 1.f / D;
  // with WPR > 1 every warp of the block runs the same number of iterations (barriers inside row_sum)
  const long long stride = (long long)gridDim.x * RPB;
  const long long first = (long long)blockIdx.x * RPB;
  for (long long base = first; base < rows; base += stride) {
    long long row = base + row_in_block;
    const bool live = row < rows;
    if (WPR == 1 && !live) break;
    if (!live) row = rows - 1;
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * D);
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + row * D);
    // the other gradient too where registers allow: behind the sums its latency would stand alone
    constexpr bool EARLY = sizeof(T) == 2 && VPL <= 3;
    uint4 xraw[VPL], draw[VPL], oraw[EARLY ? VPL : 1];
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int i = t + k * 32 * WPR;
      xraw[k] = i < nvec ? __ldg(xr + i) : make_uint4(0, 0, 0, 0);
      draw[k] = i < nvec ? __ldg(dyr + i) : make_uint4(0, 0, 0, 0);
      if (EARLY && dres != nullptr && i < nvec) oraw[EARLY ? k : 0] = __ldg(reinterpret_cast<const uint4*>(dres + row * D) + i);
    }
    const float mu = rms ? 0.f : mean[row];
    const float rs = rstd[row];
    const float keep = live ? 1.f : 0.f;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      if (t + k * 32 * WPR < nvec) {
        float xv[VN], dv[VN], gv[VN];
        nv_unpack<T>(xraw[k], xv);
        nv_unpack<T>(draw[k], dv);
        if (gamma) load_params<VN>(gamma, (t + k * 32 * WPR) * VN, gv);
#pragma unroll
        for (int j = 0; j < VN; ++j) {
          const float xhat = (xv[j] - mu) * rs;
          const float g = gamma ? gv[j] * dv[j] : dv[j];
          s1 += g;
          s2 += g * xhat;
          dg[k * VN + j] += keep * dv[j] * xhat;
          db[k * VN + j] += keep * dv[j];
        }
      }
    }
    const float m2 = row_sum<NT, WPR>(s2, red, row_in_block, warp_in_row, lane, 0) * inv_d;
    const float m1 = rms ? 0.f : row_sum<NT, WPR>(s1, red, row_in_block, warp_in_row, lane, 1) * inv_d;
    if (WPR > 1 && rms) __syncthreads();  // keep the two-phase alternation of `red` when the second reduction is skipped
    if (live) {
      uint4* dxr = reinterpret_cast<uint4*>(dx + row * D);
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int i = t + k * 32 * WPR;
        if (i < nvec) {
          float xv[VN], dv[VN], gv[VN];
          nv_unpack<T>(xraw[k], xv);
          nv_unpack<T>(draw[k], dv);
          if (gamma) load_params<VN>(gamma, i * VN, gv);
#pragma unroll
          for (int j = 0; j < VN; ++j) {
            const float xhat = (xv[j] - mu) * rs;
            const float g = gamma ? gv[j] * dv[j] : dv[j];
            dv[j] = rs * (g - m1 - xhat * m2);
          }
          if (dres != nullptr) {  // what reaches the normalised sum on its other way
            float ov[VN];
            nv_unpack<T>(EARLY ? oraw[EARLY ? k : 0] : __ldg(reinterpret_cast<const uint4*>(dres + row * D) + i), ov);
#pragma unroll
            for (int j = 0; j < VN; ++j) dv[j] += ov[j];
          }
          dxr[i] = nv_pack<T>(dv);
        }
      }
    }
  }
  // reduction over the block's row groups, one quantity at a time through shared memory
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    float* out = pass == 0 ? partial_dgamma : partial_dbeta;
    if (out == nullptr) continue;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < VPL; ++k)
#pragma unroll
      for (int j = 0; j < VN; ++j) {
        const int c = (t + k * 32 * WPR) * VN + j;
        if (c < D) nsm[row_in_block * D + c] = pass == 0 ? dg[k * VN + j] : db[k * VN + j];
      }
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += NT) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < RPB; ++w) s += nsm[w * D + c];
      out[(long long)blockIdx.x * D + c] = s;
    }
  }
}

// Sums `nblocks` partial rows of D columns: 32 columns x 32 row groups per block, four loads in flight per thread.
__global__ void __launch_bounds__(1024) norm_partial_reduce2_kernel(const float* __restrict__ pa, float* __restrict__ oa, const float* __restrict__ pb,
                                                                    float* __restrict__ ob, int nblocks, int D, int accumulate) {
  __shared__ float tile[32][33];
  const float* partial = blockIdx.y == 0 ? pa : pb;
  float* out = blockIdx.y == 0 ? oa : ob;
  if (partial == nullptr || out == nullptr) return;
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  if (c < D) {
    int b = ry;
    for (; b + 96 < nblocks; b += 128) {
      s0 += partial[(long long)b * D + c];
      s1 += partial[(long long)(b + 32) * D + c];
      s2 += partial[(long long)(b + 64) * D + c];
      s3 += partial[(long long)(b + 96) * D + c];
    }
    for (; b < nblocks; b += 32) s0 += partial[(long long)b * D + c];
  }
  tile[ry][cx] = (s0 + s1) + (s2 + s3);
  __syncthreads();
  if (ry == 0 && c < D) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 32; ++r) s += tile[r][cx];
    out[c] = accumulate ? out[c] + s : s;
  }
}

// rms != 0: RMSNorm (no mean subtraction, no beta)
template <typename T>
__global__ void __launch_bounds__(NORM_THREADS) norm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ res, T* __restrict__ sum_out, const float* __restrict__ gamma,
                                                                const float* __restrict__ beta,
                                                                T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int D,
                                                                float eps, int rms, int narrow) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const T* xr = x + row * D;
  auto value = [&](int i) { return res != nullptr ? to_f32<T>(from_f32<T>(to_f32<T>(xr[i]) + to_f32<T>(res[row * D + i]))) : to_f32<T>(xr[i]); };
  T* yr = y + row * D;
  float s = 0.f, ss = 0.f;
  for (int i = threadIdx.x; i < D; i += NORM_THREADS) {
    const float v = value(i);
    if (res != nullptr) sum_out[row * D + i] = from_f32<T>(v);
    s += v;
    ss += v * v;
  }
  s = block_sum(s, red);
  ss = block_sum(ss, red);
  const float mean = rms ? 0.f : s / D;
  const float var = rms ? ss / D : fmaxf(ss / D - mean * mean, 0.f);
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
  for (int i = threadIdx.x; i < D; i += NORM_THREADS) {
    float v = (value(i) - mean) * rstd;
    if (gamma) v *= narrow ? to_f32<T>(from_f32<T>(gamma[i])) : gamma[i];
    if (beta) v += narrow ? to_f32<T>(from_f32<T>(beta[i])) : beta[i];
    yr[i] = from_f32<T>(v);
  }
}

// Each block walks rows blockIdx.x, +gridDim.x, ...; thread t owns columns t, t+256, ... (<= MAXC per thread)
template <typename T, int MAXC>
__global__ void __launch_bounds__(NORM_THREADS) norm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ gamma,
                                                                const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ dres,
                                                                T* __restrict__ dx, float* __restrict__ partial_dgamma, float* __restrict__ partial_dbeta,
                                                                long long rows, int D, int rms) {
  __shared__ float red[32];
  float dg[MAXC], db[MAXC];
#pragma unroll
  for (int k = 0; k < MAXC; ++k) { dg[k] = 0.f; db[k] = 0.f; }
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* xr = x + row * D;
    const T* dyr = dy + row * D;
    const float mu = rms ? 0.f : mean[row];
    const float rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < MAXC; ++k) {
      const int i = threadIdx.x + k * NORM_THREADS;
      if (i < D) {
        const float xhat = (to_f32<T>(xr[i]) - mu) * rs;
        const float d = to_f32<T>(dyr[i]);
        const float g = gamma ? gamma[i] * d : d;
        s1 += g;
        s2 += g * xhat;
        dg[k] += d * xhat;
        db[k] += d;
      }
    }
    s1 = block_sum(s1, red);
    s2 = block_sum(s2, red);
    const float m1 = rms ? 0.f : s1 / D, m2 = s2 / D;
    T* dxr = dx + row * D;
#pragma unroll
    for (int k = 0; k < MAXC; ++k) {
      const int i = threadIdx.x + k * NORM_THREADS;
      if (i < D) {
        const float xhat = (to_f32<T>(xr[i]) - mu) * rs;
        const float d = to_f32<T>(dyr[i]);
        const float g = gamma ? gamma[i] * d : d;
        dxr[i] = from_f32<T>(rs * (g - m1 - xhat * m2) + (dres != nullptr ? to_f32<T>(dres[row * D + i]) : 0.f));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < MAXC; ++k) {
    const int i = threadIdx.x + k * NORM_THREADS;
    if (i < D) {
      partial_dgamma[(long long)blockIdx.x * D + i] = dg[k];
      if (partial_dbeta) partial_dbeta[(long long)blockIdx.x * D + i] = db[k];
    }
  }
}

__global__ void norm_partial_reduce_kernel(const float* __restrict__ partial, float* __restrict__ out, int nblocks, int D, int accumulate) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= D) return;
  float s = 0.f;
  for (int b = 0; b < nblocks; ++b) s += partial[(long long)b * D + i];
  out[i] = accumulate ? out[i] + s : s;
}

// y = norm(x), or norm(sum) with sum = x + res where `res` is given: a block of a transformer adds its branch and normalises the sum, and
// the sum has another reader, the next addition; one pass writes both.  [16384, 768] bf16: 10.7 + 13.5 us apart, 16.6 together.
// mean / rstd: null where nobody takes a gradient.  narrow: gamma and beta are rounded to the type of the rows as they are read.
KB_API int kb200_norm_fwd(const void* x, const void* res, void* sum, const float* gamma, const float* beta, void* y, float* mean, float* rstd, long long rows, int D,
                          float eps, int rms, int narrow, int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  {
    const int vn = dtype == 1 ? 8 : 4;
    const bool aligned = ((((uintptr_t)x | (uintptr_t)res | (uintptr_t)sum | (uintptr_t)y | (uintptr_t)gamma | (uintptr_t)beta) & 15) == 0) && D % vn == 0;
    const int nvec = aligned ? D / vn : 0;
    // shapes: (threads, warps per row); up to 8 vectors per thread
#define LAUNCH_FW(T, VPL, NT, WPR)                                                                                                                \
  do {                                                                                                                                            \
    constexpr int rpb = NT / 32 / WPR;                                                                                                            \
    norm_fwd_warp_kernel<T, VPL, NT, WPR><<<(unsigned)((rows + rpb - 1) / rpb), NT, 0, stream>>>((const T*)x, (const T*)res, (T*)sum, gamma, beta, (T*)y, mean, rstd, \
                                                                                                  rows, D, eps, rms, narrow);                     \
  } while (0)
#define PICK_FW(T)                                                   \
  do {                                                               \
    if (nvec <= 32) LAUNCH_FW(T, 1, 128, 1);                         \
    else if (nvec <= 64) LAUNCH_FW(T, 2, 128, 1);                    \
    else if (nvec <= 96) LAUNCH_FW(T, 3, 128, 1);                    \
    else if (nvec <= 128) LAUNCH_FW(T, 4, 128, 1);                   \
    else if (nvec <= 256) LAUNCH_FW(T, 2, 128, 4);                   \
    else if (nvec <= 512) LAUNCH_FW(T, 4, 128, 4);                   \
    else if (nvec <= 1024) LAUNCH_FW(T, 4, 256, 8);                  \
    else LAUNCH_FW(T, 8, 256, 8);                                    \
  } while (0)
    if (nvec >= 1 && nvec <= 2048) {
      if (dtype == 1) PICK_FW(__nv_bfloat16);
      else PICK_FW(float);
      KB_CHECK_LAUNCH("norm_fwd");
      return 0;
    }
#undef PICK_FW
#undef LAUNCH_FW
  }
  if (dtype == 1)
    norm_fwd_kernel<__nv_bfloat16><<<(unsigned)rows, NORM_THREADS, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (__nv_bfloat16*)sum, gamma, beta, (__nv_bfloat16*)y, mean, rstd, D, eps, rms, narrow);
  else
    norm_fwd_kernel<float><<<(unsigned)rows, NORM_THREADS, 0, stream>>>((const float*)x, (const float*)res, (float*)sum, gamma, beta, (float*)y, mean, rstd, D, eps, rms, narrow);
  KB_CHECK_LAUNCH("norm_fwd");
  return 0;
}

KB_API int kb200_norm_bwd_blocks(long long rows) {
  long long b = 148 * 6;
  return (int)(rows < b ? rows : b);
}

// partial_dgamma / partial_dbeta: scratch [kb200_norm_bwd_blocks(rows), D] fp32; accumulate != 0: dgamma and dbeta are added to
// `dres`: a gradient of x from elsewhere that is added to dx (of a residual sum, whose other reader is the next addition), or null.
KB_API int kb200_norm_bwd(const void* dy, const void* x, const float* gamma, const float* mean, const float* rstd, const void* dres, void* dx, float* partial_dgamma,
                          float* partial_dbeta, float* dgamma, float* dbeta, long long rows, int D, int rms, int dtype, int accumulate,
                          cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D > NORM_THREADS * 32) { kb200_set_error("norm_bwd: D too large (max 8192)"); return -2; }
  int blocks = kb200_norm_bwd_blocks(rows);
  {
    const int vn = dtype == 1 ? 8 : 4;
    const bool aligned = ((((uintptr_t)x | (uintptr_t)dy | (uintptr_t)dx | (uintptr_t)dres | (uintptr_t)gamma) & 15) == 0) && D % vn == 0;
    const int nvec = aligned ? D / vn : 0;
#define LAUNCH_BW(T, VPL, NT, WPR, ...)                                                                                                            \
  do {                                                                                                                                             \
    const size_t smem = (size_t)(NT / 32 / WPR) * D * sizeof(float);                                                                               \
    norm_bwd_warp_kernel<T, VPL, NT, WPR, ##__VA_ARGS__><<<blocks, NT, smem, stream>>>((const T*)dy, (const T*)x, gamma, mean, rstd, (const T*)dres, (T*)dx, partial_dgamma,      \
                                                                         partial_dbeta, rows, D, rms);                                             \
  } while (0)
    // per-thread accumulators: 2 x VPL x (8 or 4) floats, so at most 4 vectors per thread for bf16 and 8 for fp32
    bool done = true;
    if (dtype == 1) {
      const int resident = (nvec > 64 ? 3 : 4) * kb_sm_count();  // what runs at once below 1024 columns: a second, shorter wave would only add partial sums
      if (nvec >= 1 && nvec <= 96 && blocks > resident) blocks = resident;
      if (nvec < 1) done = false;
      else if (nvec <= 32) LAUNCH_BW(__nv_bfloat16, 1, 128, 1, 4);
      else if (nvec <= 64) LAUNCH_BW(__nv_bfloat16, 2, 128, 1, 4);
      else if (nvec <= 96) LAUNCH_BW(__nv_bfloat16, 3, 128, 1, 3);
      else if (nvec <= 128) LAUNCH_BW(__nv_bfloat16, 4, 128, 1, 3);
      else if (nvec <= 256) LAUNCH_BW(__nv_bfloat16, 2, 128, 4);
      else if (nvec <= 512) LAUNCH_BW(__nv_bfloat16, 4, 128, 4);
      else if (nvec <= 1024) LAUNCH_BW(__nv_bfloat16, 4, 256, 8);
      else done = false;
    } else {
      if (nvec < 1) done = false;
      else if (nvec <= 32) LAUNCH_BW(float, 1, 128, 1);
      else if (nvec <= 64) LAUNCH_BW(float, 2, 128, 1);
      else if (nvec <= 128) LAUNCH_BW(float, 4, 128, 1);
      else if (nvec <= 256) LAUNCH_BW(float, 8, 128, 1);
      else if (nvec <= 512) LAUNCH_BW(float, 4, 128, 4);
      else if (nvec <= 1024) LAUNCH_BW(float, 8, 128, 4);
      else if (nvec <= 2048) LAUNCH_BW(float, 8, 256, 8);
      else done = false;
    }
#undef LAUNCH_BW
    if (done) {
      KB_CHECK_LAUNCH("norm_bwd");
      if (dgamma || (dbeta && partial_dbeta)) {
        dim3 grid((D + 31) / 32, 2);
        norm_partial_reduce2_kernel<<<grid, 1024, 0, stream>>>(dgamma ? partial_dgamma : nullptr, dgamma, partial_dbeta, dbeta, blocks, D, accumulate);
        KB_CHECK_LAUNCH("norm_partial_reduce");
      }
      return 0;
    }
  }
  const int per = (D + NORM_THREADS - 1) / NORM_THREADS;
#define LAUNCH(T, MAXC)                                                                                                            \
  norm_bwd_kernel<T, MAXC><<<blocks, NORM_THREADS, 0, stream>>>((const T*)dy, (const T*)x, gamma, mean, rstd, (const T*)dres, (T*)dx, partial_dgamma, \
                                                                 partial_dbeta, rows, D, rms)
  if (dtype == 1) {
    if (per <= 4) LAUNCH(__nv_bfloat16, 4);
    else if (per <= 8) LAUNCH(__nv_bfloat16, 8);
    else if (per <= 16) LAUNCH(__nv_bfloat16, 16);
    else LAUNCH(__nv_bfloat16, 32);
  } else {
    if (per <= 4) LAUNCH(float, 4);
    else if (per <= 8) LAUNCH(float, 8);
    else if (per <= 16) LAUNCH(float, 16);
    else LAUNCH(float, 32);
  }
#undef LAUNCH
  KB_CHECK_LAUNCH("norm_bwd");
  if (dgamma) norm_partial_reduce_kernel<<<(D + 127) / 128, 128, 0, stream>>>(partial_dgamma, dgamma, blocks, D, accumulate);
  if (dbeta && partial_dbeta) norm_partial_reduce_kernel<<<(D + 127) / 128, 128, 0, stream>>>(partial_dbeta, dbeta, blocks, D, accumulate);
  KB_CHECK_LAUNCH("norm_partial_reduce");
  return 0;
}

// ---------------------------------------------------------------------------------------------
// Column sums of a [rows, cols] bf16/fp32 matrix into fp32 (bias gradients): blocks of 32 column vectors x 8 row lanes
// accumulate a slab of rows in registers, combine the row lanes through shared memory and write one partial row per
// slab; norm_partial_reduce2_kernel sums the slabs in a fixed order.
template <typename T>
__global__ void __launch_bounds__(256) colsum_partial_kernel(const T* __restrict__ x, long long ld, long long rows, int cols, float* __restrict__ partial) {
  constexpr int VN = NVec<T>::N;
  __shared__ float sm[8][32 * VN + 1];
  const int cv = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * 32 + cv) * VN;
  const long long per = (rows + gridDim.y - 1) / gridDim.y;
  const long long r0 = (long long)blockIdx.y * per, r1 = min(rows, r0 + per);
  float acc[VN];
#pragma unroll
  for (int j = 0; j < VN; ++j) acc[j] = 0.f;
  if (c0 < cols) {
    for (long long r = r0 + rl; r < r1; r += 8) {
      float v[VN];
      nv_unpack<T>(__ldg(reinterpret_cast<const uint4*>(x + r * ld + c0)), v);
#pragma unroll
      for (int j = 0; j < VN; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < VN; ++j) sm[rl][cv * VN + j] = acc[j];
  __syncthreads();
  for (int c = threadIdx.x; c < 32 * VN; c += 256) {
    const int col = blockIdx.x * 32 * VN + c;
    if (col < cols) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) s += sm[k][c];
      partial[(long long)blockIdx.y * cols + col] = s;
    }
  }
}

// dz = dy * act'(z) and, in the same pass, the column sums of dz (the bias gradient of the layer in front): three tensors moved where
// the library's derivative and a separate sum move four.  [16384, 3072] gelu: 83 + 20 -> 73 us; the traffic takes 45.
// A ReLU selects instead of multiplying: an infinite gradient at a closed one is nothing, and one at a NaN passes, as in the library.
enum { AB_RELU = 1, AB_SILU = 3, AB_GELU = 4 };
template <int ACT>
__device__ __forceinline__ float act_grad(float z) {
  if (ACT == AB_SILU) {
    const float s = 1.f / (1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
  }
  return fmaf(z * 0.3989422804014327f, __expf(-0.5f * z * z), normal_cdf(z));
}

template <int ACT>
__global__ void __launch_bounds__(256) act_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ z,
                                                      __nv_bfloat16* __restrict__ dz, long long rows, int cols, float* __restrict__ partial) {
  constexpr int VN = 8, U = 2;
  __shared__ float sm[8][32 * VN + 1];
  const int cv = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * 32 + cv) * VN;
  const long long per = (rows + gridDim.y - 1) / gridDim.y;
  const long long r0 = (long long)blockIdx.y * per, r1 = min(rows, r0 + per);
  float acc[VN] = {};
  if (c0 < cols) {
    for (long long r = r0 + rl; r < r1; r += 8 * U) {
      uint4 g[U], q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r + 8 * u < r1) {
          g[u] = *reinterpret_cast<const uint4*>(dy + (r + 8 * u) * cols + c0);
          q[u] = *reinterpret_cast<const uint4*>(z + (r + 8 * u) * cols + c0);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r + 8 * u >= r1) continue;
        float gv[VN], zv[VN];
        unpack8(reinterpret_cast<const bf16x8&>(g[u]), gv);
        unpack8(reinterpret_cast<const bf16x8&>(q[u]), zv);
#pragma unroll
        for (int j = 0; j < VN; ++j) gv[j] = ACT == AB_RELU ? (zv[j] <= 0.f ? 0.f : gv[j]) : gv[j] * act_grad<ACT>(zv[j]);
        const bf16x8 out = pack8(gv);
        *reinterpret_cast<bf16x8*>(dz + (r + 8 * u) * cols + c0) = out;
        unpack8(out, gv);  // the sum is that of the values as stored
#pragma unroll
        for (int j = 0; j < VN; ++j) acc[j] += gv[j];
      }
    }
  }
  if (partial == nullptr) return;
#pragma unroll
  for (int j = 0; j < VN; ++j) sm[rl][cv * VN + j] = acc[j];
  __syncthreads();
  for (int c = threadIdx.x; c < 32 * VN; c += 256) {
    const int col = blockIdx.x * 32 * VN + c;
    if (col < cols) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) s += sm[k][c];
      partial[(long long)blockIdx.y * cols + col] = s;
    }
  }
}

// out[c] = sum over the rows of partial [slabs, cols], added to what out holds where `accumulate`; a fixed order
KB_API int kb200_sum_slabs(const float* partial, float* out, int slabs, int cols, int accumulate, cudaStream_t stream) {
  if (cols <= 0) return 0;
  norm_partial_reduce2_kernel<<<dim3((cols + 31) / 32, 1), 1024, 0, stream>>>(partial, out, nullptr, nullptr, slabs, cols, accumulate);
  KB_CHECK_LAUNCH("sum_slabs");
  return 0;
}

KB_API int kb200_colsum_slabs(long long rows, int cols, int dtype) {
  const int vn = dtype == 1 ? 8 : 4;
  const int col_blocks = (cols + 32 * vn - 1) / (32 * vn);
  long long slabs = (148 * 6 + col_blocks - 1) / col_blocks;
  if (slabs > (rows + 63) / 64) slabs = (rows + 63) / 64;
  if (slabs < 1) slabs = 1;
  if (slabs > 512) slabs = 512;
  return (int)slabs;
}

// x: [rows, cols] with row pitch ld (elements), cols a multiple of the 16-byte vector and rows 16-byte aligned;
// partial: scratch [kb200_colsum_slabs(rows, cols, dtype), cols] fp32; out: [cols] fp32.
// accumulate != 0: out += the sums (a bias gradient added into persistent storage).
KB_API int kb200_colsum(const void* x, long long ld, long long rows, int cols, float* partial, float* out, int dtype, int accumulate,
                        cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  const int vn = dtype == 1 ? 8 : 4;
  if (cols % vn || ld % vn || ((uintptr_t)x & 15)) {
    kb200_set_error("colsum: columns and pitch must be multiples of the 16-byte vector and the base pointer aligned");
    return -2;
  }
  const int slabs = kb200_colsum_slabs(rows, cols, dtype);
  dim3 grid((cols + 32 * vn - 1) / (32 * vn), slabs);
  if (dtype == 1)
    colsum_partial_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, ld, rows, cols, partial);
  else
    colsum_partial_kernel<float><<<grid, 256, 0, stream>>>((const float*)x, ld, rows, cols, partial);
  KB_CHECK_LAUNCH("colsum");
  dim3 grid2((cols + 31) / 32, 1);
  norm_partial_reduce2_kernel<<<grid2, 1024, 0, stream>>>(partial, out, nullptr, nullptr, slabs, cols, accumulate);
  KB_CHECK_LAUNCH("colsum_reduce");
  return 0;
}

// normal_cdf with one more coefficient (fit and float32 as there, t = 1 / (1 + 0.4 a): 7e-8; 4.5e-7 of the lower tail for a < 1 and 5.5e-7 for a < 2, 3.5e-7
// of the upper one), where a pass is bound by its traffic anyway.
__device__ __forceinline__ float normal_cdf_near(float v) {
  const float a = fabsf(v), t = __fdividef(1.f, fmaf(0.4f, a, 1.f)), x = a * 0.8493218002880191f;
  float p = 0.27416810393333435f;
  p = fmaf(p, t, -1.4040862321853638f);
  p = fmaf(p, t, 2.8040099143981934f);
  p = fmaf(p, t, -2.5186238288879395f);
  p = fmaf(p, t, 0.7767177224159241f);
  p = fmaf(p, t, -0.2595641016960144f);
  p = fmaf(p, t, 0.536329448223114f);
  p = fmaf(p, t, 1.43856942653656f);
  p = fmaf(p, t, -2.6475203037261963f);
  const float lower = t * exp2f(fmaf(-x, x, p));
  return v > 0.f ? 1.f - lower : lower;
}

// y = gelu(z), exact, bf16: the activation behind a product whose input the backward pass needs as it was.  Bound by its traffic: four
// vectors a thread in flight, and a normal distribution function of seventeen instructions.  [16384, 3072] 59 us (the library's) -> 37; 201 MB take 31.
// Before the rounding a value is within 5.4e-7 for z > -2 (the library's 1 + erff: 1.0e-6; 4.7e-7 and 1.2e-7 for z > 0) and 3.1e-6 below, where that one
// has lost all digits at z = -6.  After it the two are equally far from 64 bits, 1.729824e-3 over 5e7 normal values, and differ in that tail alone.
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const uint4* __restrict__ z, uint4* __restrict__ y, long long vecs) {
  constexpr int U = 4;
  const long long first = (long long)blockIdx.x * 256 * U + threadIdx.x;
  uint4 raw[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (first + u * 256 < vecs) raw[u] = __ldg(z + first + u * 256);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (first + u * 256 < vecs) {
      float v[8];
      nv_unpack<__nv_bfloat16>(raw[u], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= normal_cdf_near(v[j]);
      y[first + u * 256] = nv_pack<__nv_bfloat16>(v);
    }
  }
}

// n values, a multiple of 8, 16-byte aligned
KB_API int kb200_gelu_fwd(const void* z, void* y, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8 || (((uintptr_t)z | (uintptr_t)y) & 15) || n / 8192 > 0x7ffffff0ll) {
    kb200_set_error("gelu_fwd: values in multiples of 8, 16-byte aligned");
    return -2;
  }
  gelu_fwd_kernel<<<(unsigned)((n + 8191) / 8192), 256, 0, stream>>>((const uint4*)z, (uint4*)y, n / 8);
  KB_CHECK_LAUNCH("gelu_fwd");
  return 0;
}

// dz = dy * act'(z) on contiguous bf16 [rows, cols] (cols a multiple of 8, 16-byte aligned bases), act: 1 relu, 3 silu, 4 gelu (erf).
// With partial (scratch as for kb200_colsum) the column sums of dz go to out, or are added to it (accumulate).
KB_API int kb200_act_bwd(const void* dy, const void* z, void* dz, long long rows, int cols, int act, float* partial, float* out, int accumulate,
                         cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return 0;
  if (cols % 8 || (((uintptr_t)dy | (uintptr_t)z | (uintptr_t)dz) & 15) || (act != AB_RELU && act != AB_SILU && act != AB_GELU)) {
    kb200_set_error("act_bwd: columns must be a multiple of 8, bases aligned, the activation relu, silu or gelu");
    return -2;
  }
  const int slabs = kb200_colsum_slabs(rows, cols, 1);
  dim3 grid((cols + 255) / 256, slabs);
  const __nv_bfloat16 *g = (const __nv_bfloat16*)dy, *q = (const __nv_bfloat16*)z;
  if (act == AB_RELU) act_bwd_kernel<AB_RELU><<<grid, 256, 0, stream>>>(g, q, (__nv_bfloat16*)dz, rows, cols, partial);
  else if (act == AB_SILU) act_bwd_kernel<AB_SILU><<<grid, 256, 0, stream>>>(g, q, (__nv_bfloat16*)dz, rows, cols, partial);
  else act_bwd_kernel<AB_GELU><<<grid, 256, 0, stream>>>(g, q, (__nv_bfloat16*)dz, rows, cols, partial);
  KB_CHECK_LAUNCH("act_bwd");
  if (partial != nullptr) {
    norm_partial_reduce2_kernel<<<dim3((cols + 31) / 32, 1), 1024, 0, stream>>>(partial, out, nullptr, nullptr, slabs, cols, accumulate);
    KB_CHECK_LAUNCH("act_bwd_reduce");
  }
  return 0;
}
