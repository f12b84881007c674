// Depthwise 2-D convolution of channels-last bf16 tensors, depth multiplier 1: y[n, oh, ow, c] = sum_rs x[n, oh*S - pt + r, ow*S - pl + s, c] w[r, s, c],
// its data gradient and its weight gradient.  Square filters of 3, 5 or 7 taps, stride 1 or 2 (the same in both directions); padding is a
// matter of coordinates, so no padded copy is made.  Replaces the grouped library convolution behind
// keras/src/backend/torch/nn.py:717-760 and the layout and padding copies around it.
//
// Every pass is bound by its tensors' traffic (9 to 49 multiply-adds a value).  A thread owns 8 channels (one 16-byte vector) and a
// strip of 4 pixels of a row: a row of input vectors is loaded once, all loads in flight together, unpacked once and used for every
// pixel of the strip; the rows above and below come from L1 / L2, where the neighbouring strips left them.  Sums are fp32 in a fixed
// order; the weight gradient sums strips per thread, then per CTA, then over the CTAs' partial sums, each time in a fixed order, so that it
// is the same bit for bit from run to run (an atomic add per CTA and weight took 55 us where this takes 60 at 56x56x144 and stride 2, 40 / 45 at
// 28x28x192, 62 / 66 with 5x5 there).
// The lanes of a warp take whole pixels side by side (dw_grid) and two channels share a multiply-add instruction: at stride 2, 56x56x144,
// forward 65 -> 42 us, data gradient 80 -> 52, weight gradient 78 -> 58; 28x28x192 at stride 1 37 -> 35, 37 -> 35, 49 -> 42; 5x5 there
// 66 -> 61, 66 -> 61, 87 -> 64 (the weight gradients with atomics).  (A thread that walks down its strip and keeps three rows of sums, 196 registers, was no quicker: 37 us.)
// us, this / the library (which pads and re-lays in passes of its own at stride 2), 128 images:
//   56x56x144 3x3 /2   forward 42 / 208   both gradients 114 / 395     28x28x192 5x5   forward 61 / 66   gradients 129 / 230
//   28x28x192 3x3      forward 35 / 31    both gradients  82 / 121     56x56x96 7x7 (64 images)   109 / 115   257 / 673
#include "common.cuh"

extern "C" int kb200_sum_slabs(const float* partial, float* out, int slabs, int cols, int accumulate, cudaStream_t stream);

namespace {

constexpr int TW = 4, TW2 = 2, THREADS = 256;  // pixels of a strip; TW2: data gradient at stride 2

struct DwArgs {
  const __nv_bfloat16* x;   // forward, weight gradient: input;  data gradient: dy
  const __nv_bfloat16* w;   // [K, K, C]
  __nv_bfloat16* y;         // forward: output;  data gradient: dx
  const __nv_bfloat16* dy;  // weight gradient
  float* partial;           // weight gradient: [gridDim.x][K, K, C]
  int N, H, W, C, OH, OW, pt, pl;
  int cx;                   // channel vectors of a CTA
};

// Two floats in a 64-bit register: one fused multiply-add does both (each rounded as by itself).
using f2 = unsigned long long;
__device__ __forceinline__ uint4 load_vec(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ f2 pair_of(uint32_t u) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(u << 16), "r"(u & 0xffff0000u));
  return d;
}
__device__ __forceinline__ void unpack_vec(const uint4& r, f2* f) {
  f[0] = pair_of(r.x), f[1] = pair_of(r.y), f[2] = pair_of(r.z), f[3] = pair_of(r.w);
}
__device__ __forceinline__ void fma2(f2& acc, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint32_t pack_pair(f2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return reinterpret_cast<const uint32_t&>(b);
}
__device__ __forceinline__ void store_vec(__nv_bfloat16* p, const f2* v) {
  *reinterpret_cast<uint4*>(p) = make_uint4(pack_pair(v[0]), pack_pair(v[1]), pack_pair(v[2]), pack_pair(v[3]));
}
// Weights in shared memory, as floats: [taps][half of a vector][32 vectors][4].  Channels side by side give no bank conflicts, and a
// pitch known here makes every address an immediate.
constexpr int SW_HALF = 32 * 4, SW_TAP = 2 * SW_HALF;
__device__ __forceinline__ void load_tap(const float* sw, f2* w) {
  *reinterpret_cast<ulonglong2*>(w) = *reinterpret_cast<const ulonglong2*>(sw);
  *reinterpret_cast<ulonglong2*>(w + 2) = *reinterpret_cast<const ulonglong2*>(sw + SW_HALF);
}

// Stage the CTA's weights.  FLIP: the taps in reverse order (data gradient at stride 1).
template <int K, bool FLIP>
__device__ __forceinline__ void stage_weights(const DwArgs& a, float* sw, int cvec0, int cx) {
  const int ch = cx * 8;
  for (int i = threadIdx.x; i < K * K * ch; i += THREADS) {
    const int tap = i / ch, at = i % ch, c = cvec0 * 8 + at;
    sw[tap * SW_TAP + (at >> 2 & 1) * SW_HALF + (at >> 3) * 4 + (at & 3)] =
        c < a.C ? __bfloat162float(a.w[(size_t)(FLIP ? K * K - 1 - tap : tap) * a.C + c]) : 0.f;
  }
  __syncthreads();
}

// FLIP = false: forward.  FLIP = true (stride 1): data gradient, the same sum with mirrored taps; the launcher mirrors the padding.
template <int K, int S, bool FLIP>
__global__ void __launch_bounds__(THREADS, 2) depthwise_kernel(const DwArgs a) {
  extern __shared__ float sw[];
  const int cx = a.cx, cvecs = a.C / 8, per = THREADS / cx, slot = threadIdx.x / cx;
  const int tx = threadIdx.x - slot * cx, cv = blockIdx.y * cx + tx;
  stage_weights<K, FLIP>(a, sw, blockIdx.y * cx, cx);
  if (cv >= cvecs || slot >= per) return;
  const unsigned strips = (a.OW + TW - 1) / TW;
  const unsigned total = (unsigned)(a.N * a.OH * strips), step = gridDim.x * per;
  constexpr int IN = (TW - 1) * S + K;
  for (unsigned t = blockIdx.x * per + slot; t < total; t += step) {
    const unsigned line = t / strips;  // 32-bit divisions: the launcher keeps the pixels below 2^30
    const int ow0 = (int)(t - line * strips) * TW, oh = (int)(line % a.OH);
    const long long n = line / a.OH;
    const int iw0 = ow0 * S - a.pl, ih0 = oh * S - a.pt;
    f2 acc[TW][4] = {};
#pragma unroll
    for (int r = 0; r < K; ++r) {
      const int ih = ih0 + r;
      if ((unsigned)ih >= (unsigned)a.H) continue;
      const __nv_bfloat16* row = a.x + ((n * a.H + ih) * a.W + iw0) * a.C + cv * 8;
      uint4 raw[IN];
#pragma unroll
      for (int i = 0; i < IN; ++i) raw[i] = (unsigned)(iw0 + i) < (unsigned)a.W ? load_vec(row + (long long)i * a.C) : make_uint4(0, 0, 0, 0);
      f2 w[K][4];
#pragma unroll
      for (int s = 0; s < K; ++s) load_tap(sw + (r * K + s) * SW_TAP + tx * 4, w[s]);
#pragma unroll
      for (int i = 0; i < IN; ++i) {
        f2 v[4];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = i - j * S;
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 4; ++e) fma2(acc[j][e], v[e], w[s][e]);
          }
        }
      }
    }
    __nv_bfloat16* out = a.y + ((n * a.OH + oh) * a.OW + ow0) * a.C + cv * 8;
#pragma unroll
    for (int j = 0; j < TW; ++j)
      if (ow0 + j < a.OW) store_vec(out + (long long)j * a.C, acc[j]);
  }
}

// Strips of 2 with 64 registers (four CTAs an SM) hide the latency of the few loads a strip has better than strips of 4: [128, 56, 56,
// 144] 3x3 116 -> 81 us, 5x5 152 -> 126 (before the lanes took whole pixels).
// Data gradient at stride 2: dx[ih, iw] = sum dy[oh, ow] w[ih + pt - 2 oh, iw + pl - 2 ow].  Strips start where iw + pl is even, so that the
// taps of each pixel are known at compile time.
template <int K>
__global__ void __launch_bounds__(THREADS, 4) depthwise_dgrad2_kernel(const DwArgs a) {
  extern __shared__ float sw[];
  constexpr int S = 2, TW = TW2;
  const int cx = a.cx, cvecs = a.C / 8, per = THREADS / cx, slot = threadIdx.x / cx;
  const int tx = threadIdx.x - slot * cx, cv = blockIdx.y * cx + tx;
  stage_weights<K, false>(a, sw, blockIdx.y * cx, cx);
  if (cv >= cvecs || slot >= per) return;
  const int off = a.pl & 1;
  const unsigned strips = (a.W + off + TW - 1) / TW;
  const unsigned total = (unsigned)(a.N * a.H * strips), step = gridDim.x * per;
  constexpr int BACK = (K - 1) / S, COLS = BACK + (TW - 1) / S + 1;  // output columns base/2 - BACK ... base/2 + (TW - 1)/2
  for (unsigned t = blockIdx.x * per + slot; t < total; t += step) {
    const unsigned line = t / strips;
    const int iw0 = (int)(t - line * strips) * TW - off, ih = (int)(line % a.H);
    const long long n = line / a.H;
    const int ow0 = (iw0 + a.pl) / S - BACK;
    f2 acc[TW][4] = {};
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
      f2 w[K][4];
#pragma unroll
      for (int s = 0; s < K; ++s) load_tap(sw + (r * K + s) * SW_TAP + tx * 4, w[s]);
#pragma unroll
      for (int i = 0; i < COLS; ++i) {
        f2 v[4];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = j - S * (i - BACK);
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 4; ++e) fma2(acc[j][e], v[e], w[s][e]);
          }
        }
      }
    }
    __nv_bfloat16* out = a.y + ((n * a.H + ih) * a.W + iw0) * a.C + cv * 8;
#pragma unroll
    for (int j = 0; j < TW; ++j)
      if ((unsigned)(iw0 + j) < (unsigned)a.W) store_vec(out + (long long)j * a.C, acc[j]);
  }
}

// R rows of taps a thread (all of them for 3x3, whose 72 sums fit the registers; else one, blockIdx.z): dw[r, s] += x[oh*S - pt + r, ow*S - pl + s] dy[oh, ow]
template <int K, int S, int R>
__global__ void __launch_bounds__(THREADS, K == 5 ? 2 : 1) depthwise_wgrad_kernel(const DwArgs a) {
  __shared__ float red[THREADS * 8];
  const int cx = a.cx, cvecs = a.C / 8, per = THREADS / cx, slot = threadIdx.x / cx;
  const int tx = threadIdx.x - slot * cx, cv = blockIdx.y * cx + tx;
  const int r_first = blockIdx.z * R;
  const bool active = cv < cvecs && slot < per;
  const unsigned strips = (a.OW + TW - 1) / TW;
  const unsigned total = active ? (unsigned)(a.N * a.OH * strips) : 0u, step = gridDim.x * per;
  constexpr int IN = (TW - 1) * S + K;
  f2 acc[R][K][4] = {};
  for (unsigned t = blockIdx.x * per + slot; t < total; t += step) {
    const unsigned line = t / strips;
    const int ow0 = (int)(t - line * strips) * TW, oh = (int)(line % a.OH);
    const long long n = line / a.OH;
    const int iw0 = ow0 * S - a.pl;
    const __nv_bfloat16* grow = a.dy + ((n * a.OH + oh) * a.OW + ow0) * a.C + cv * 8;
    f2 g[TW][4];
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
        f2 v[4];
        unpack_vec(raw[i], v);
#pragma unroll
        for (int j = 0; j < TW; ++j) {
          const int s = i - j * S;
          if (s >= 0 && s < K) {
#pragma unroll
            for (int e = 0; e < 4; ++e) fma2(acc[r][s][e], v[e], g[j][e]);
          }
        }
      }
    }
  }
  // one tap at a time: the CTA's threads hand their sums over, cx * 8 channels times `groups` threads add them up, then the groups' sums
  const int lanes = cx * 8, groups = THREADS / lanes, group = threadIdx.x / lanes, ci = threadIdx.x - group * lanes;
  const int c = blockIdx.y * lanes + ci;
  float* out = a.partial + (size_t)blockIdx.x * K * K * a.C;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < K; ++s) {
      __syncthreads();
      *reinterpret_cast<ulonglong2*>(red + threadIdx.x * 8) = make_ulonglong2(acc[r][s][0], acc[r][s][1]);
      *reinterpret_cast<ulonglong2*>(red + threadIdx.x * 8 + 4) = make_ulonglong2(acc[r][s][2], acc[r][s][3]);
      __syncthreads();
      float sum = 0.f;
      if (group < groups)
        for (int i = group; i < per; i += groups) sum += red[i * lanes + ci];
      if (groups > 1) {
        __syncthreads();
        red[threadIdx.x] = sum;
        __syncthreads();
        if (group == 0)
          for (int g = 1; g < groups; ++g) sum += red[g * lanes + ci];
      }
      if (group == 0 && c < a.C) out[(size_t)((r_first + r) * K + s) * a.C + c] = sum;
    }
}

struct DwGrid {
  dim3 grid;
  int cx;
};

// Channel vectors of a CTA: eight (128 bytes, whole lines, and few distinct weights a warp) where that divides them, else an even share of
// at most 32, so that a warp reads pixels whole.  (A power of two that divides 18 vectors is 2: 32 bytes of each pixel, and an L1 that
// found 31 % of the sectors that are read again.)  The weight gradient has no weights to read and takes the share always.
DwGrid dw_grid(int C, long long strips, int ctas_per_sm, int z, bool eights) {
  const int cvecs = C / 8;
  DwGrid g;
  g.cx = (cvecs + (cvecs + 31) / 32 - 1) / ((cvecs + 31) / 32);
  if (eights && cvecs % 8 == 0) g.cx = 8;
  const int gy = (cvecs + g.cx - 1) / g.cx;
  const int per = THREADS / g.cx;
  long long gx = (strips + per - 1) / per, cap = (long long)kb_sm_count() * ctas_per_sm / ((long long)gy * z);
  if (cap < 1) cap = 1;
  if (gx > cap) gx = cap;
  g.grid = dim3((unsigned)gx, (unsigned)gy, (unsigned)z);
  return g;
}

long long out_strips(int N, int OH, int OW) { return (long long)N * OH * ((OW + TW - 1) / TW); }

DwGrid wgrad_grid(int N, int OH, int OW, int C, int K) { return dw_grid(C, out_strips(N, OH, OW), 2, K == 3 ? 1 : K, false); }

template <int K>
int dw_launch(int mode, DwArgs a, int S, cudaStream_t st) {
  const long long in_strips = (long long)a.N * a.H * ((a.W + 1 + TW2 - 1) / TW2);
  const DwGrid g = mode == 0   ? dw_grid(a.C, out_strips(a.N, a.OH, a.OW), 16, 1, true)
                   : mode == 1 ? dw_grid(a.C, in_strips, 16, 1, true)
                               : wgrad_grid(a.N, a.OH, a.OW, a.C, K);
  a.cx = g.cx;
  const int smem = mode == 2 ? 0 : K * K * SW_TAP * 4;
  if (smem > 48 * 1024) {  // 7x7: 49 KB and more
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

// Partial sums of a weight gradient: the first dimension of `partial` below.
KB_API int kb200_depthwise_slabs(int N, int OH, int OW, int C, int K) {
  return N <= 0 || OH <= 0 || OW <= 0 || C < 8 || K <= 0 ? 0 : (int)wgrad_grid(N, OH, OW, C, K).grid.x;
}

// mode 0: y = conv(x, w);  1: y = dx from x = dy;  2: dw (fp32) from x and dy, added to what dw holds where `accumulate`; partial: scratch, fp32
// [kb200_depthwise_slabs, K, K, C].  x: [N, H, W, C], dy: [N, OH, OW, C], w: [K, K, C]; C a multiple of 8, 16-byte aligned bases.
// (pt, pl): rows and columns of zeros in front of the input.
KB_API int kb200_depthwise(int mode, const void* x, const void* w, void* y, const void* dy, float* dw, float* partial, int accumulate, int N, int H, int W, int C,
                           int OH, int OW, int K, int S, int pt, int pl, cudaStream_t stream) {
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
  DwArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (const __nv_bfloat16*)dy, partial, N, H, W, C, OH, OW, pt, pl, 0};
  const int rc = K == 3 ? dw_launch<3>(mode, a, S, stream) : K == 5 ? dw_launch<5>(mode, a, S, stream) : dw_launch<7>(mode, a, S, stream);
  if (rc != 0) return rc;
  KB_CHECK_LAUNCH("depthwise");
  return mode == 2 ? kb200_sum_slabs(partial, dw, kb200_depthwise_slabs(N, OH, OW, C, K), K * K * C, accumulate, stream) : 0;
}
