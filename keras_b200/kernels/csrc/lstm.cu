// A whole LSTM layer in one launch a direction: every time step of z_t = x_t W (+ b) + h_{t-1} R, its gates and its state, float32.
//
//   i, f, o = sigmoid(z_i, z_f, z_o)   g = tanh(z_g)   c_t = f c_{t-1} + i g   h_t = o tanh(c_t)
//
// The projection x W of all steps is one product made by the caller.  What is left is a chain: step by step it was a dozen small
// kernels forward and two dozen backward, each waiting for the one before (keras/src/layers/rnn/lstm.py:240-300 under a loop).
//
// Here each CTA owns 16 units (their four gates) for a group of batch rows and keeps its slice of R in shared memory for the whole
// sequence, so a step moves only the state: 8 rows of h in (32 KB of gradients backward at 256 units), 16 columns of h out.  The
// CTAs of one row group exchange h through L2 and meet at a counter after each step; groups never wait for one another.  Row
// tiles of 8 keep that exchange small, which is what bounds a step at the usual sizes (latency of L2 and of the counter), and the
// fp32 FMA rate bounds it at the largest.  Products and sums are plain fp32; the K range is split over the warps and summed in a
// fixed order, so results do not depend on timing.
//
// 64 rows x 100 steps x 256 units, 32 features: training step 10.4 -> 1.38 ms (4146 -> 56 launches in its graph), of which 428 us
// forward and 555 us backward in these kernels, 4.3 and 5.6 us a step.
//
// The launch is cooperative (all CTAs resident).  Every wait is bounded: on expiry the kernel records a code in *err and returns.
#include "common.cuh"

namespace {

constexpr int UNITS = 16, ROWS = 8, COLS = 4 * UNITS, THREADS = 256, WARPS = THREADS / 32;
constexpr int KC = 1024;          // backward: columns of dz staged at a time
constexpr int MAX_UNITS = 640;    // 256 bytes of R a unit stay within shared memory
constexpr uint32_t SPIN_LIMIT = 1u << 22;

struct LstmArgs {
  const float* xz;       // [B, T, 4U], time index t
  const float* bias;     // [4U] or null
  const float* h0;       // [B, U]
  const float* c0;       // [B, U]
  const float* R;        // [U, 4U]
  float* hprev;          // [B, T, U]: the state that enters step t
  float* out;            // [B, T, U] in processing order, or null
  float* hT;             // [B, U]
  float* cT;             // [B, U]
  float* gates;          // [T, B, 4U] after their activations, processing order; null without gradients
  float* cs;             // [T, B, U], processing order; with gates
  // backward
  const float* dout;     // [B, T, U] or null
  const float* dhT;      // [B, U] or null
  const float* dcT;      // [B, U] or null
  float* dz;             // [B, T, 4U], time index t
  float* dh0;            // [B, U] or null
  float* dc0;            // [B, U]: workspace of the running gradient of c, in the end that of c0
  int* counters;         // one per row group, zero on entry
  int* err;
  int B, T, U, reverse, slices, rows_per_group;
};

__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ bool meet(int* counter, int target, int* flag, int* err) {
  // all threads call; true when every CTA of the group has arrived `target / slices` times
  if (threadIdx.x == 0) {
    int ok = 0;
    for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
      int v;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) {
        ok = 1;
        break;
      }
    }
    if (!ok) atomicExch(err, 41);
    *flag = ok;
  }
  __syncthreads();
  return *flag != 0;
}

__device__ __forceinline__ void arrive(int* counter) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(counter) : "memory");
  }
}

__global__ void __launch_bounds__(THREADS, 1) lstm_forward_kernel(const LstmArgs a) {
  extern __shared__ float smem[];
  __shared__ int flag;
  const int U = a.U, T = a.T, B = a.B, pitch = U + 4;
  float* Rs = smem;                       // [U][64]: gate-major columns of this CTA's units
  float* hs = Rs + (size_t)U * COLS;      // [8][U + 4]
  float* part = hs + ROWS * pitch;        // [8 warps][8 rows][64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x % a.slices, group = blockIdx.x / a.slices;
  const int u0 = slice * UNITS, nu = min(UNITS, U - u0);
  const int row_begin = group * a.rows_per_group, row_end = min(B, row_begin + a.rows_per_group);
  int* counter = a.counters + group;

  for (int i = tid; i < U * COLS; i += THREADS) {
    const int k = i / COLS, j = i % COLS, u = j % UNITS;
    Rs[i] = u < nu ? a.R[(size_t)k * 4 * U + (j / UNITS) * U + u0 + u] : 0.f;
  }
  const int cg = (lane & 15) * 4, rg = (lane >> 4) * 4;
  const int prow = (tid & 127) / UNITS, pu = tid % UNITS;  // pointwise part: threads 0..127, one (row, unit) each
  float bias[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) bias[g] = a.bias != nullptr && pu < nu ? a.bias[g * U + u0 + pu] : 0.f;
  bool ok = true;

  for (int p = 0; p < T && ok; ++p) {
    const int t = a.reverse ? T - 1 - p : p;
    for (int r0 = row_begin; r0 < row_end; r0 += ROWS) {
      const int row = r0 + prow;
      const bool mine = tid < 128 && row < row_end && pu < nu;
      float z[4] = {0.f, 0.f, 0.f, 0.f}, c = 0.f;
      if (mine) {  // independent of the other CTAs: in flight while this one waits for them
        const float* x = a.xz + ((size_t)row * T + t) * 4 * U + u0 + pu;
#pragma unroll
        for (int g = 0; g < 4; ++g) z[g] = x[(size_t)g * U] + bias[g];
        c = p == 0 ? a.c0[(size_t)row * U + u0 + pu]
                   : a.gates != nullptr ? a.cs[((size_t)(p - 1) * B + row) * U + u0 + pu] : a.cT[(size_t)row * U + u0 + pu];
      }
      if (p > 0 && r0 == row_begin) {
        ok = meet(counter, p * a.slices, &flag, a.err);
        if (!ok) break;
      }
      for (int i = tid; i < ROWS * (U / 4); i += THREADS) {
        const int r = i / (U / 4), k = (i % (U / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + r < row_end) {
          const float* src = p == 0 ? a.h0 + (size_t)(r0 + r) * U : a.hprev + ((size_t)(r0 + r) * T + t) * U;
          v = __ldcg(reinterpret_cast<const float4*>(src + k));  // written by other CTAs: past L1
        }
        *reinterpret_cast<float4*>(hs + r * pitch + k) = v;
      }
      __syncthreads();
      float acc[4][4] = {};
      for (int k = warp * 4; k < U; k += WARPS * 4) {
        float4 h[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) h[r] = *reinterpret_cast<const float4*>(hs + (rg + r) * pitch + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(Rs + (size_t)(k + i) * COLS + cg);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float v = i == 0 ? h[r].x : i == 1 ? h[r].y : i == 2 ? h[r].z : h[r].w;
            acc[r][0] += v * w.x;
            acc[r][1] += v * w.y;
            acc[r][2] += v * w.z;
            acc[r][3] += v * w.w;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4*>(part + (warp * ROWS + rg + r) * COLS + cg) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      __syncthreads();
      if (mine) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float s = 0.f;
#pragma unroll
          for (int w = 0; w < WARPS; ++w) s += part[(w * ROWS + prow) * COLS + g * UNITS + pu];
          z[g] += s;
        }
        const float gi = sigmoid_f(z[0]), gf = sigmoid_f(z[1]), gg = tanhf(z[2]), go = sigmoid_f(z[3]);
        c = gf * c + gi * gg;
        const float h = go * tanhf(c);
        const size_t at = (size_t)row * U + u0 + pu;
        if (p == 0) a.hprev[((size_t)row * T + t) * U + u0 + pu] = a.h0[at];
        if (p + 1 < T) a.hprev[((size_t)row * T + (a.reverse ? t - 1 : t + 1)) * U + u0 + pu] = h;
        if (a.out != nullptr) a.out[((size_t)row * T + p) * U + u0 + pu] = h;
        if (a.gates != nullptr) {
          float* gs = a.gates + ((size_t)p * B + row) * 4 * U + u0 + pu;
          gs[0] = gi;
          gs[(size_t)U] = gf;
          gs[(size_t)2 * U] = gg;
          gs[(size_t)3 * U] = go;
          a.cs[((size_t)p * B + row) * U + u0 + pu] = c;
        }
        if (a.gates == nullptr || p + 1 == T) a.cT[at] = c;
        if (p + 1 == T) a.hT[at] = h;
      }
    }
    if (ok && p + 1 < T) arrive(counter);
  }
}

__global__ void __launch_bounds__(THREADS, 1) lstm_backward_kernel(const LstmArgs a) {
  extern __shared__ float smem[];
  __shared__ int flag;
  const int U = a.U, T = a.T, B = a.B, K = 4 * U, pitch = KC + 4;
  float* Rt = smem;                          // R^T of this CTA's units, K x 16, laid out for the lanes' order below
  float* ds = Rt + (size_t)K * UNITS;        // [8][KC + 4]
  float* part = ds + ROWS * pitch;           // [32 K slices][8 rows][16]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x % a.slices, group = blockIdx.x / a.slices;
  const int u0 = slice * UNITS, nu = min(UNITS, U - u0);
  const int row_begin = group * a.rows_per_group, row_end = min(B, row_begin + a.rows_per_group);
  int* counter = a.counters + group;

  // Blocks of 16 k; a warp's four lane groups take four k each.  k = 16 b + 4 s + i sits at b * 256 + i * 64 + s * 16, so that the
  // groups' reads for one i are 64 consecutive floats.
  for (int i = tid; i < K * UNITS; i += THREADS) {
    const int u = i / K, k = i % K;
    Rt[(k >> 4) * 256 + (k & 3) * 64 + ((k >> 2) & 3) * 16 + u] = u < nu ? a.R[(size_t)(u0 + u) * K + k] : 0.f;
  }
  const int cg = (lane & 3) * 4, rg = ((lane >> 2) & 1) * 4, ks = lane >> 3;
  const int prow = (tid & 127) / UNITS, pu = tid % UNITS;
  bool ok = true;

  const int last = a.dh0 != nullptr ? -1 : 0;  // step -1 only carries the gradient on to h0
  for (int q = T - 1; q >= last && ok; --q) {
    const int t = a.reverse ? T - 1 - q : q, t_next = a.reverse ? t - 1 : t + 1;  // t_next: time index of step q + 1
    for (int r0 = row_begin; r0 < row_end; r0 += ROWS) {
      const int row = r0 + prow;
      const bool mine = tid < 128 && row < row_end && pu < nu;
      const size_t at = (size_t)row * U + u0 + pu;
      float gi = 0.f, gf = 0.f, gg = 0.f, go = 0.f, c = 0.f, cp = 0.f, dh = 0.f, dc = 0.f;
      if (mine) {
        if (q >= 0) {
          const float* gs = a.gates + ((size_t)q * B + row) * 4 * U + u0 + pu;
          gi = gs[0];
          gf = gs[(size_t)U];
          gg = gs[(size_t)2 * U];
          go = gs[(size_t)3 * U];
          c = a.cs[((size_t)q * B + row) * U + u0 + pu];
          cp = q > 0 ? a.cs[((size_t)(q - 1) * B + row) * U + u0 + pu] : a.c0[at];
          if (a.dout != nullptr) dh = a.dout[((size_t)row * T + q) * U + u0 + pu];
        }
        if (q == T - 1) {
          if (a.dhT != nullptr) dh += a.dhT[at];
          if (a.dcT != nullptr) dc = a.dcT[at];
        } else {
          dc = a.dc0[at];  // written by this thread one step ago
        }
      }
      if (q < T - 1) {
        if (r0 == row_begin) {
          ok = meet(counter, (T - 1 - q) * a.slices, &flag, a.err);
          if (!ok) break;
        }
        float acc[4][4] = {};
        for (int k0 = 0; k0 < K; k0 += KC) {
          const int kc = min(KC, K - k0);
          for (int i = tid; i < ROWS * (kc / 4); i += THREADS) {
            const int r = i / (kc / 4), k = (i % (kc / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r0 + r < row_end) v = __ldcg(reinterpret_cast<const float4*>(a.dz + ((size_t)(r0 + r) * T + t_next) * K + k0 + k));
            *reinterpret_cast<float4*>(ds + r * pitch + k) = v;
          }
          __syncthreads();
          for (int b = warp; b < kc / 16; b += WARPS) {
            float4 d[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) d[r] = *reinterpret_cast<const float4*>(ds + (rg + r) * pitch + b * 16 + ks * 4);
            const float* w0 = Rt + (size_t)(k0 / 16 + b) * 256 + ks * 16 + cg;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 w = *reinterpret_cast<const float4*>(w0 + i * 64);
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                const float v = i == 0 ? d[r].x : i == 1 ? d[r].y : i == 2 ? d[r].z : d[r].w;
                acc[r][0] += v * w.x;
                acc[r][1] += v * w.y;
                acc[r][2] += v * w.z;
                acc[r][3] += v * w.w;
              }
            }
          }
          __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
          *reinterpret_cast<float4*>(part + ((warp * 4 + ks) * ROWS + rg + r) * UNITS + cg) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        __syncthreads();
        if (mine) {
          float s = 0.f;
#pragma unroll
          for (int w = 0; w < 32; ++w) s += part[(w * ROWS + prow) * UNITS + pu];
          dh += s;
        }
      }
      if (mine) {
        if (q >= 0) {
          const float tc = tanhf(c);
          dc += dh * go * (1.f - tc * tc);
          float* d = a.dz + ((size_t)row * T + t) * K + u0 + pu;
          d[0] = dc * gg * gi * (1.f - gi);
          d[(size_t)U] = dc * cp * gf * (1.f - gf);
          d[(size_t)2 * U] = dc * gi * (1.f - gg * gg);
          d[(size_t)3 * U] = dh * tc * go * (1.f - go);
          a.dc0[at] = dc * gf;
        } else {
          a.dh0[at] = dh;
        }
      }
    }
    if (ok && q > last) arrive(counter);
  }
}

size_t lstm_smem(int U, bool backward) {
  const size_t r = (size_t)U * COLS * 4;
  return backward ? r + ROWS * (KC + 4) * 4 + 32 * ROWS * UNITS * 4 : r + ROWS * (U + 4) * 4 + WARPS * ROWS * COLS * 4;
}
}  // namespace

// Row groups of a launch (the length of `counters`), or 0 when the kernel does not take the layer.
KB_API int kb200_lstm_groups(int B, int U) {
  if (B <= 0 || U <= 0 || U % 4 || U > MAX_UNITS) return 0;
  const int slices = (U + UNITS - 1) / UNITS, fit = kb_sm_count() / slices, tiles = (B + ROWS - 1) / ROWS;
  if (fit < 1) return 0;
  const int per = (tiles + fit - 1) / fit;  // row tiles of a group
  return (tiles + per - 1) / per;
}

KB_API int kb200_lstm(int backward, const float* xz, const float* bias, const float* h0, const float* c0, const float* R, float* hprev, float* out, float* hT,
                      float* cT, float* gates, float* cs, const float* dout, const float* dhT, const float* dcT, float* dz, float* dh0, float* dc0,
                      int* counters, int* err, int B, int T, int U, int reverse, cudaStream_t stream) {
  const int groups = kb200_lstm_groups(B, U);
  if (groups == 0 || T <= 0) {
    kb200_set_error("lstm: units must be a multiple of 4 and at most 640, with at least one row and one step");
    return -2;
  }
  const int tiles = (B + ROWS - 1) / ROWS;
  LstmArgs a{xz, bias, h0, c0, R, hprev, out, hT, cT, gates, cs, dout, dhT, dcT, dz, dh0, dc0, counters, err, B, T, U, reverse,
             (U + UNITS - 1) / UNITS, (tiles + groups - 1) / groups * ROWS};
  static bool attr_f[KB_MAX_DEVICES] = {false}, attr_b[KB_MAX_DEVICES] = {false};
  const bool allowed = backward ? kb_allow_smem(lstm_backward_kernel, (int)lstm_smem(MAX_UNITS, true), attr_b)
                                : kb_allow_smem(lstm_forward_kernel, (int)lstm_smem(MAX_UNITS, false), attr_f);
  if (!allowed) {
    kb200_set_error("lstm: cannot raise the shared-memory limit of the kernel on this device");
    return -3;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.slices * groups));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = lstm_smem(U, backward != 0);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = backward ? cudaLaunchKernelEx(&cfg, lstm_backward_kernel, a) : cudaLaunchKernelEx(&cfg, lstm_forward_kernel, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    kb200_set_error(cudaGetErrorString(e));
    return -1;
  }
  KB_CHECK_LAUNCH("lstm");
  return 0;
}
