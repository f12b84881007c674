// Depthwise 2-D convolution of channels-last bf16 tensors, depth multiplier 1: y[n, oh, ow, c] = sum_rs x[n, oh*S - pt + r, ow*S - pl + s, c] w[r, s, c],
// its data gradient and its weight gradient.  Square filters of 3, 5 or 7 taps, stride 1 or 2 (the same in both directions); padding is a
// matter of coordinates, so no padded copy is made.  Replaces the grouped library convolution behind
// keras/src/backend/torch/nn.py:717-760 and the layout and padding copies around it.
//
// Every pass is bound by its tensors' traffic (9 to 49 multiply-adds a value).  A thread owns 8 channels (one 16-byte vector) and a
// strip of 4 pixels of a row: a row of input vectors is loaded once, all loads in flight together, unpacked once and used for every
// pixel of the strip; the rows above and below come from L1 / L2, where the neighbouring strips left them.  Sums are fp32 in a fixed
// order; the weight gradient sums strips per thread, then per CTA, then with one fp32 atomic add per CTA and weight.
// us, this / the library (which pads and re-lays in passes of its own at stride 2), 128 images:
//   56x56x144 3x3 /2   forward 64 / 208   both gradients 160 / 394      28x28x192 5x5   forward 67 / 66   gradients 153 / 230
//   28x28x192 3x3      forward 38 / 32    both gradients  84 / 120      56x56x96 7x7 (64 images)   119 / 115   287 / 673
#include "common.cuh"

namespace {

constexpr int TW = 4, TW2 = 2, THREADS = 256;  // pixels of a strip; TW2: data gradient at stride 2

struct DwArgs {
  const __nv_bfloat16* x;   // forward, weight gradient: input;  data gradient: dy
  const __nv_bfloat16* w;   // [K, K, C]
  __nv_bfloat16* y;         // forward: output;  data gradient: dx
  const __nv_bfloat16* dy;  // weight gradient
  float* dw;                // weight gradient, [K, K, C], added to
  int N, H, W, C, OH, OW, pt, pl;
  int cx_log2;              // channel vectors of a CTA
};

__device__ __forceinline__ uint4 load_vec(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void unpack_vec(const uint4& r, float* f) { unpack8(reinterpret_cast<const bf16x8&>(r), f); }

// Stage the CTA's weights as floats: [taps][channels of the CTA].  FLIP: the taps in reverse order (data gradient at stride 1).
template <int K, bool FLIP>
__device__ __forceinline__ void stage_weights(const DwArgs& a, float* sw, int cvec0, int cx) {
  const int ch = cx * 8;
  for (int i = threadIdx.x; i < K * K * ch; i += THREADS) {
    const int tap = i / ch, c = cvec0 * 8 + i % ch;
    sw[i] = c < a.C ? __bfloat162float(a.w[(size_t)(FLIP ? K * K - 1 - tap : tap) * a.C + c]) : 0.f;
  }
  __syncthreads();
}

// FLIP = false: forward.  FLIP = true (stride 1): data gradient, the same sum with mirrored taps; the launcher mirrors the padding.
template <int K, int S, bool FLIP>
__global__ void __launch_bounds__(THREADS, K == 3 ? 1 : 2) depthwise_kernel(const DwArgs a) {
  extern __shared__ float sw[];
  const int cx = 1 << a.cx_log2, cvecs = a.C / 8, ch = cx * 8;
  const int tx = threadIdx.x & (cx - 1), cv = blockIdx.y * cx + tx;
  stage_weights<K, FLIP>(a, sw, blockIdx.y * cx, cx);
  if (cv >= cvecs) return;
  const unsigned strips = (a.OW + TW - 1) / TW;
  const unsigned total = (unsigned)(a.N * a.OH * strips), step = gridDim.x * (THREADS >> a.cx_log2);
  constexpr int IN = (TW - 1) * S + K;
  for (unsigned t = blockIdx.x * (THREADS >> a.cx_log2) + (threadIdx.x >> a.cx_log2); t < total; t += step) {
    const unsigned line = t / strips;  // 32-bit divisions: the launcher keeps the pixels below 2^30
    const int ow0 = (int)(t - line * strips) * TW, oh = (int)(line % a.OH);
    const long long n = line / a.OH;
    const int iw0 = ow0 * S - a.pl, ih0 = oh * S - a.pt;
    float acc[TW][8] = {};
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int ih = ih0 + r;
      if ((unsigned)ih >= (unsigned)a.H) continue;
      const __nv_bfloat16* row = a.x + ((n * a.H + ih) * a.W + iw0) * a.C + cv * 8;
      uint4 raw[IN];
#pragma unroll
      for (int i = 0; i < IN; ++i) raw[i] = (unsigned)(iw0 + i) < (unsigned)a.W ? load_vec(row + (long long)i * a.C) : make_uint4(0, 0, 0, 0);
      float w[K][8];
#pragma unroll
      for (int s = 0; s < K; ++s) {
        *reinterpret_cast<float4*>(w[s]) = *reinterpret_cast<const float4*>(sw + (r * K + s) * ch + tx * 8);
        *reinterpret_cast<float4*>(w[s] + 4) = *reinterpret_cast<const float4*>(sw + (r * K + s) * ch + tx * 8 + 4);
      }
#pragma unroll
      for (int i = 0; i < IN; ++i) {
        float v[8];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = i - j * S;
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[j][e] += v[e] * w[s][e];
          }
        }
      }
    }
    __nv_bfloat16* out = a.y + ((n * a.OH + oh) * a.OW + ow0) * a.C + cv * 8;
#pragma unroll
    for (int j = 0; j < TW; ++j)
      if (ow0 + j < a.OW) *reinterpret_cast<bf16x8*>(out + (long long)j * a.C) = pack8(acc[j]);
  }
}

// Strips of 2 with 64 registers (four CTAs an SM) hide the latency of the few loads a strip has better than strips of 4: [128, 56, 56,
// 144] 3x3 116 -> 81 us, 5x5 152 -> 126.
// Data gradient at stride 2: dx[ih, iw] = sum dy[oh, ow] w[ih + pt - 2 oh, iw + pl - 2 ow].  Strips start where iw + pl is even, so that the
// taps of each pixel are known at compile time.
template <int K>
__global__ void __launch_bounds__(THREADS, 4) depthwise_dgrad2_kernel(const DwArgs a) {
  extern __shared__ float sw[];
  constexpr int S = 2, TW = TW2;
  const int cx = 1 << a.cx_log2, cvecs = a.C / 8, ch = cx * 8;
  const int tx = threadIdx.x & (cx - 1), cv = blockIdx.y * cx + tx;
  stage_weights<K, false>(a, sw, blockIdx.y * cx, cx);
  if (cv >= cvecs) return;
  const int off = a.pl & 1;
  const unsigned strips = (a.W + off + TW - 1) / TW;
  const unsigned total = (unsigned)(a.N * a.H * strips), step = gridDim.x * (THREADS >> a.cx_log2);
  constexpr int BACK = (K - 1) / S, COLS = BACK + (TW - 1) / S + 1;  // output columns base/2 - BACK ... base/2 + (TW - 1)/2
  for (unsigned t = blockIdx.x * (THREADS >> a.cx_log2) + (threadIdx.x >> a.cx_log2); t < total; t += step) {
    const unsigned line = t / strips;
    const int iw0 = (int)(t - line * strips) * TW - off, ih = (int)(line % a.H);
    const long long n = line / a.H;
    const int ow0 = (iw0 + a.pl) / S - BACK;
    float acc[TW][8] = {};
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int hh = ih + a.pt - r;
      if (hh & 1) continue;
      const int oh = hh >> 1;  // floor: a negative one stays negative
      if ((unsigned)oh >= (unsigned)a.OH) continue;
      const __nv_bfloat16* row = a.x + ((n * a.OH + oh) * a.OW + ow0) * a.C + cv * 8;
      uint4 raw[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) raw[i] = (unsigned)(ow0 + i) < (unsigned)a.OW ? load_vec(row + (long long)i * a.C) : make_uint4(0, 0, 0, 0);
      float w[K][8];
#pragma unroll
      for (int s = 0; s < K; ++s) {
        *reinterpret_cast<float4*>(w[s]) = *reinterpret_cast<const float4*>(sw + (r * K + s) * ch + tx * 8);
        *reinterpret_cast<float4*>(w[s] + 4) = *reinterpret_cast<const float4*>(sw + (r * K + s) * ch + tx * 8 + 4);
      }
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        float v[8];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = j - S * (i - BACK);
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[j][e] += v[e] * w[s][e];
          }
        }
      }
    }
    __nv_bfloat16* out = a.y + ((n * a.H + ih) * a.W + iw0) * a.C + cv * 8;
#pragma unroll
    for (int j = 0; j < TW; ++j)
      if ((unsigned)(iw0 + j) < (unsigned)a.W) *reinterpret_cast<bf16x8*>(out + (long long)j * a.C) = pack8(acc[j]);
  }
}

// R rows of taps a thread (all of them for 3x3, whose 72 sums fit the registers; else one, blockIdx.z): dw[r, s] += x[oh*S - pt + r, ow*S - pl + s] dy[oh, ow]
template <int K, int S, int R>
__global__ void __launch_bounds__(THREADS, K == 3 ? 1 : 2) depthwise_wgrad_kernel(const DwArgs a) {
  extern __shared__ float red[];  // [THREADS / cx strips] folded to warps: [8 warps][cx * 8]
  const int cx = 1 << a.cx_log2, cvecs = a.C / 8;
  const int tx = threadIdx.x & (cx - 1), cv = blockIdx.y * cx + tx;
  const int r_first = blockIdx.z * R;
  const bool active = cv < cvecs;
  const unsigned strips = (a.OW + TW - 1) / TW;
  const unsigned total = active ? (unsigned)(a.N * a.OH * strips) : 0u, step = gridDim.x * (THREADS >> a.cx_log2);
  constexpr int IN = (TW - 1) * S + K;
  float acc[R][K][8] = {};
  for (unsigned t = blockIdx.x * (THREADS >> a.cx_log2) + (threadIdx.x >> a.cx_log2); t < total; t += step) {
    const unsigned line = t / strips;
    const int ow0 = (int)(t - line * strips) * TW, oh = (int)(line % a.OH);
    const long long n = line / a.OH;
    const int iw0 = ow0 * S - a.pl;
    const __nv_bfloat16* grow = a.dy + ((n * a.OH + oh) * a.OW + ow0) * a.C + cv * 8;
    float g[TW][8];
#pragma unroll
    for (int j = 0; j < TW; ++j) unpack_vec(ow0 + j < a.OW ? load_vec(grow + (long long)j * a.C) : make_uint4(0, 0, 0, 0), g[j]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ih = oh * S - a.pt + r_first + r;
      if ((unsigned)ih >= (unsigned)a.H) continue;
      const __nv_bfloat16* row = a.x + ((n * a.H + ih) * a.W + iw0) * a.C + cv * 8;
      uint4 raw[IN];
#pragma unroll
      for (int i = 0; i < IN; ++i) raw[i] = (unsigned)(iw0 + i) < (unsigned)a.W ? load_vec(row + (long long)i * a.C) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < IN; ++i) {
        float v[8];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = i - j * S;
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[r][s][e] += v[e] * g[j][e];
          }
        }
      }
    }
  }
  // threads of a warp that own the same channels differ by multiples of cx; then the warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < K; ++s) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        for (int o = 16; o >= cx; o >>= 1) acc[r][s][e] += __shfl_xor_sync(0xffffffffu, acc[r][s][e], o);
      __syncthreads();
      if (lane < cx) {
#pragma unroll
        for (int e = 0; e < 8; ++e) red[(warp * cx + lane) * 8 + e] = acc[r][s][e];
      }
      __syncthreads();
      for (int i = threadIdx.x; i < cx * 8; i += THREADS) {
        const int c = blockIdx.y * cx * 8 + i;
        if (c < a.C) {
          float sum = 0.f;
#pragma unroll
          for (int w = 0; w < THREADS / 32; ++w) sum += red[w * cx * 8 + i];
          atomicAdd(a.dw + (size_t)((r_first + r) * K + s) * a.C + c, sum);
        }
      }
    }
}

struct DwGrid {
  dim3 grid;
  int cx_log2;
};

// Channel vectors of a CTA: the power of two up to 32 that wastes the fewest threads; CTAs along the pixels: `waves` residencies at most.
DwGrid dw_grid(int C, long long strips, int ctas_per_sm, int z) {
  const int cvecs = C / 8;
  int best = 0;
  long long least = -1;
  for (int l = 0; l <= 5; ++l) {
    const long long lanes = (long long)((cvecs + (1 << l) - 1) >> l) << l;
    if (least < 0 || lanes <= least) {
      least = lanes;
      best = l;
    }
  }
  DwGrid g;
  g.cx_log2 = best;
  const int gy = (cvecs + (1 << best) - 1) >> best, per = THREADS >> best;
  long long gx = (strips + per - 1) / per, cap = (long long)kb_sm_count() * ctas_per_sm / ((long long)gy * z);
  if (cap < 1) cap = 1;
  if (gx > cap) gx = cap;
  g.grid = dim3((unsigned)gx, (unsigned)gy, (unsigned)z);
  return g;
}

template <int K>
int dw_launch(int mode, DwArgs a, int S, cudaStream_t st) {
  const long long out_strips = (long long)a.N * a.OH * ((a.OW + TW - 1) / TW), in_strips = (long long)a.N * a.H * ((a.W + 1 + TW2 - 1) / TW2);
  const DwGrid g = mode == 0 ? dw_grid(a.C, out_strips, 16, 1) : mode == 1 ? dw_grid(a.C, in_strips, 16, 1) : dw_grid(a.C, out_strips, 2, K == 3 ? 1 : K);
  a.cx_log2 = g.cx_log2;
  const int smem = mode == 2 ? (THREADS / 32) * (1 << a.cx_log2) * 8 * 4 : K * K * (1 << a.cx_log2) * 8 * 4;
  if (smem > 48 * 1024) {  // 7x7 with 32 vectors: 50 KB
    static bool f1[KB_MAX_DEVICES] = {false}, f2[KB_MAX_DEVICES] = {false}, b1[KB_MAX_DEVICES] = {false}, b2[KB_MAX_DEVICES] = {false};
    if (!kb_allow_smem(depthwise_kernel<K, 1, false>, smem, f1) || !kb_allow_smem(depthwise_kernel<K, 2, false>, smem, f2) ||
        !kb_allow_smem(depthwise_kernel<K, 1, true>, smem, b1) || !kb_allow_smem(depthwise_dgrad2_kernel<K>, smem, b2)) {
      kb200_set_error("depthwise: cannot raise the shared-memory limit of the kernel on this device");
      return -3;
    }
  }
  if (mode == 0) {
    if (S == 1) depthwise_kernel<K, 1, false><<<g.grid, THREADS, smem, st>>>(a);
    else depthwise_kernel<K, 2, false><<<g.grid, THREADS, smem, st>>>(a);
  } else if (mode == 1) {
    if (S == 1) {  // dx = dy convolved with the mirrored filter
      DwArgs m = a;
      m.H = a.OH; m.W = a.OW; m.OH = a.H; m.OW = a.W;
      m.pt = K - 1 - a.pt; m.pl = K - 1 - a.pl;
      depthwise_kernel<K, 1, true><<<g.grid, THREADS, smem, st>>>(m);
    } else {
      depthwise_dgrad2_kernel<K><<<g.grid, THREADS, smem, st>>>(a);
    }
  } else {
    constexpr int R = K == 3 ? 3 : 1;
    if (S == 1) depthwise_wgrad_kernel<K, 1, R><<<g.grid, THREADS, smem, st>>>(a);
    else depthwise_wgrad_kernel<K, 2, R><<<g.grid, THREADS, smem, st>>>(a);
  }
  return 0;
}
}  // namespace

// mode 0: y = conv(x, w);  1: y = dx from x = dy;  2: dw (fp32, added to) from x and dy.  x: [N, H, W, C], dy: [N, OH, OW, C], w: [K, K, C]; C a multiple
// of 8, 16-byte aligned bases.  (pt, pl): rows and columns of zeros in front of the input.
KB_API int kb200_depthwise(int mode, const void* x, const void* w, void* y, const void* dy, float* dw, int N, int H, int W, int C, int OH, int OW, int K, int S,
                           int pt, int pl, cudaStream_t stream) {
  if (N <= 0 || H <= 0 || W <= 0 || C <= 0 || OH <= 0 || OW <= 0) return 0;
  if ((long long)N * H * W >= (1ll << 30) || (long long)N * OH * OW >= (1ll << 30)) {
    kb200_set_error("depthwise: more than 2^30 pixels");
    return -2;
  }
  if (C % 8 || (S != 1 && S != 2) || (K != 3 && K != 5 && K != 7) || pt < 0 || pl < 0 || pt >= K || pl >= K ||
      (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y | (uintptr_t)dy) & 15)) {
    kb200_set_error("depthwise: 3, 5 or 7 taps, stride 1 or 2, channels a multiple of 8, 16-byte aligned tensors");
    return -2;
  }
  DwArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (const __nv_bfloat16*)dy, dw, N, H, W, C, OH, OW, pt, pl, 0};
  const int rc = K == 3 ? dw_launch<3>(mode, a, S, stream) : K == 5 ? dw_launch<5>(mode, a, S, stream) : dw_launch<7>(mode, a, S, stream);
  if (rc != 0) return rc;
  KB_CHECK_LAUNCH("depthwise");
  return 0;
}
