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
// forward and 555 us backward in these kernels, 4.3 and 5.6 us a step; with the clusters below, and the weight gradients by a kernel for many rows, 0.93 ms.
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

// ---------------------------------------------------------------------------------------------
// Up to 256 units the CTAs of a row group are one thread-block cluster, and the state goes from shared memory to shared memory.
//
// A step is a chain of latencies: through L2 the state takes a store, a fence, an atomic, the poll of the counter and a load, three of
// the 4.3 us of a step.  Here every CTA writes its 16 columns of h straight into the buffers of its peers (st.async), whose mbarrier counts the
// bytes: one trip.  Backward, a CTA multiplies the gate gradients of its own units by its slice of R and sends each peer that peer's
// part of the sum, a quarter of what it would take to hand out the gate gradients themselves.  The slice of R stays in registers, so
// shared memory only serves the state, as broadcasts, and two K values are multiplied an instruction.  What is left is issue slots: a
// row of a tile costs 330 cycles a step, 128 of them the products (fp32 FMA rate), the rest the gates' functions and their stores.
// Two buffers a tile suffice: a peer can send step s + 2 only after it has this CTA's part of s + 1, sent after the last read of s.
// Clusters never wait for one another, so the grid may be any size.
// 100 steps x 256 units, forward / backward: 64 rows 420 -> 290 / 554 -> 394 us, 8 rows 490 -> 153 / 680 -> 190; 64 rows x 64 units
// 340 -> 130 / 410 -> 175.  Beyond 256 units R does not fit the registers of sixteen SMs: the kernels above stay.
constexpr int CLUSTER_MAX = 16, CLUSTER_UNITS = CLUSTER_MAX * UNITS, TILES_MAX = 4;

__device__ __forceinline__ uint32_t shared_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void send4(uint32_t dst, uint32_t bar, float4 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool received(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < (SPIN_LIMIT >> 2); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float sum_of(unsigned long long v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }

// R: rows of a tile.  A tile's products take sixteen warps; the pointwise part takes one for eight units of a row.
constexpr int GEMV_WARPS = 16;
template <int R>
constexpr int cluster_threads() { return 32 * (2 * R > GEMV_WARPS ? 2 * R : GEMV_WARPS); }
template <int R>
constexpr int row_chunk() { return R == 10 ? 5 : R < 4 ? R : 4; }  // rows whose sums are in registers at a time
constexpr int padded_rows(int R) { return (R + 3) / 4 * 4; }
constexpr int DZ_GATE = UNITS + 4, DZ_ROW = 4 * DZ_GATE + 4;        // pitches that keep the lanes' reads and writes in different banks
constexpr int peer_part(int R) { return UNITS * padded_rows(R) + 8; }  // what a peer sends backward: [16 units][rows], and 32 bytes so that four peers' parts start in different banks

// KW: K values a warp multiplies, 16 KW >= U.  Grid: clusters x slices; `a.slices` CTAs a cluster, `a.rows_per_group` rows a cluster.
template <int R, int KW>
__global__ void __launch_bounds__(cluster_threads<R>(), 1) lstm_cluster_forward_kernel(const LstmArgs a) {
  constexpr int P = GEMV_WARPS * KW, THREADS = cluster_threads<R>(), RC = row_chunk<R>();  // P: row pitch of the state
  extern __shared__ float4 smem4[];
  __shared__ alignas(8) unsigned long long bars[TILES_MAX * 2];
  const int U = a.U, T = a.T, B = a.B, S = a.slices;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x % S, group = blockIdx.x / S;  // the rank in the cluster is the slice
  const int u0 = slice * UNITS, nu = min(UNITS, U - u0);
  const int row_begin = group * a.rows_per_group, row_end = min(B, row_begin + a.rows_per_group);
  const int tiles = (row_end - row_begin + R - 1) / R;
  float* hs = reinterpret_cast<float*>(smem4);                    // [tile][2][R][P]
  float* parts = hs + (size_t)(a.rows_per_group / R) * 2 * R * P;  // [2][16 warps][R][64]
  float* cs = parts + 2 * GEMV_WARPS * R * COLS;                  // [tile][THREADS]: c of this thread
  const uint32_t bytes = (uint32_t)(R * S * UNITS * 4);

  for (int i = tid; i < tiles * 2 * R * P; i += THREADS) {
    const int k = i % P, r = (i / P) % R, b = (i / P / R) & 1, row = row_begin + (i / P / R / 2) * R + r;
    hs[i] = b == 0 && k < U && row < row_end ? a.h0[(size_t)row * U + k] : 0.f;
  }
  if (tid == 0) {
    for (int i = 0; i < tiles * 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_u32(bars + i)));
      expect(shared_u32(bars + i), bytes);  // steps 1 and 2
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // A lane is one gate of one unit of eight: columns `lane` (units 0-7) and `lane + 32` (units 8-15) of the products, one of them in
  // the pointwise part, where warp w has row w / 2 and units 8 (w % 2) onwards.
  const int gate = lane >> 3;
  unsigned long long w[2][KW / 2];
  if (warp < GEMV_WARPS) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < KW; k += 2) {
        const int k0 = warp * KW + k, u = j * 8 + (lane & 7);
        const float* src = a.R + (size_t)k0 * 4 * U + (size_t)gate * U + u0 + u;
        w[j][k / 2] = pair_of(u < nu && k0 < U ? src[0] : 0.f, u < nu && k0 + 1 < U ? src[(size_t)4 * U] : 0.f);
      }
  }
  const int prow = warp >> 1, pu = (warp & 1) * 8 + (lane & 7);
  const bool pointwise = warp < 2 * R, unit_ok = pu < nu;
  const float bias = a.bias != nullptr && unit_ok ? a.bias[gate * U + u0 + pu] : 0.f;
  // where this thread reads and writes at the present step of tile 0; they move by a step at a time
  const long long step_x = a.reverse ? -4LL * U : 4LL * U, step_h = a.reverse ? -(long long)U : (long long)U, step_c = (long long)B * U;
  const long long tile_x = (long long)R * T * 4 * U, tile_h = (long long)R * T * U;
  const size_t first = (size_t)(row_begin + prow) * T + (a.reverse ? T - 1 : 0);
  const float* xp = a.xz + first * 4 * U + gate * U + u0 + pu;
  float* gp = a.gates != nullptr ? a.gates + (size_t)(row_begin + prow) * 4 * U + gate * U + u0 + pu : nullptr;
  // of the four lanes of a unit one writes the state, one c and one the output: each with its pointer, step and tile stride
  float* hp = a.hprev + first * U + u0 + pu;
  float* sp = gate == 0 ? hp + step_h : gate == 1 ? (a.gates != nullptr ? a.cs + (size_t)(row_begin + prow) * U + u0 + pu : nullptr)
                                      : gate == 2 && a.out != nullptr ? a.out + (size_t)(row_begin + prow) * T * U + u0 + pu : nullptr;
  const long long step_s = gate == 0 ? step_h : gate == 1 ? step_c : U, tile_s = gate == 1 ? (long long)R * U : tile_h;
  if (pointwise) {
    for (int i = 0; i < tiles; ++i) {
      const int row = row_begin + i * R + prow;
      const bool mine = row < row_end && unit_ok;
      cs[i * THREADS + tid] = mine ? a.c0[(size_t)row * U + u0 + pu] : 0.f;
      if (mine && gate == 0) hp[i * tile_h] = a.h0[(size_t)row * U + u0 + pu];
    }
  }
  float x = pointwise && row_begin + prow < row_end && unit_ok ? *xp : 0.f;  // the next item's projected input: a step ahead of its use
  cluster_meet();  // every peer's buffers are set and its barriers initialised

  bool ok = true;
  int item = 0;
  for (int p = 0; p < T && ok; ++p) {
    const int b = p & 1;
    for (int i = 0; i < tiles; ++i, ++item) {
      const uint32_t bar = shared_u32(bars + i * 2 + b), next_bar = shared_u32(bars + i * 2 + (b ^ 1));
      const float* h_in = hs + (size_t)(i * 2 + b) * R * P + warp * KW;
      float* part = parts + (item & 1) * GEMV_WARPS * R * COLS;  // two: a tile's sums are still read while the next one's are written
      if (warp < GEMV_WARPS) {
        if (p > 0) ok = received(bar, (uint32_t)((p - 1) >> 1) & 1u);
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += RC) {
          unsigned long long acc[RC][2];
#pragma unroll
          for (int r = 0; r < RC; ++r) acc[r][0] = acc[r][1] = 0ull;
#pragma unroll
          for (int k = 0; k < KW / 4; ++k) {
#pragma unroll
            for (int r = 0; r < RC; ++r) {
              const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(h_in + (r0 + r) * P + k * 4);
              acc[r][0] = fma2(h.x, w[0][2 * k], acc[r][0]);
              acc[r][1] = fma2(h.x, w[1][2 * k], acc[r][1]);
              acc[r][0] = fma2(h.y, w[0][2 * k + 1], acc[r][0]);
              acc[r][1] = fma2(h.y, w[1][2 * k + 1], acc[r][1]);
            }
          }
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            part[(warp * R + r0 + r) * COLS + lane] = sum_of(acc[r][0]);
            part[(warp * R + r0 + r) * COLS + lane + 32] = sum_of(acc[r][1]);
          }
        }
      }
      ok = __syncthreads_and(ok);
      if (!ok) break;
      if (tid == 0 && p > 0 && p + 2 < T) expect(bar, bytes);  // every thread is past this phase
      if (pointwise) {
        const bool mine = row_begin + i * R + prow < row_end && unit_ok;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int v = 0; v < GEMV_WARPS; ++v) s[v & 3] += part[(v * R + prow) * COLS + (warp & 1) * 32 + lane];
        const float z = x + bias + ((s[0] + s[1]) + (s[2] + s[3]));
        const float act = gate == 2 ? tanhf(z) : sigmoid_f(z);
        const int l8 = lane & 7;
        const float gi = __shfl_sync(0xffffffffu, act, l8), gf = __shfl_sync(0xffffffffu, act, 8 + l8);
        const float gg = __shfl_sync(0xffffffffu, act, 16 + l8), go = __shfl_sync(0xffffffffu, act, 24 + l8);
        const float c = gf * cs[i * THREADS + tid] + gi * gg;
        const float h = unit_ok ? go * tanhf(c) : 0.f;
        if (p + 1 < T) {
          const int chunk = (lane & 1) * 4, peer = lane >> 1;
          float4 v;
          v.x = __shfl_sync(0xffffffffu, h, chunk);
          v.y = __shfl_sync(0xffffffffu, h, chunk + 1);
          v.z = __shfl_sync(0xffffffffu, h, chunk + 2);
          v.w = __shfl_sync(0xffffffffu, h, chunk + 3);
          if (peer < S) {
            const uint32_t dst = shared_u32(hs + ((size_t)(i * 2 + (b ^ 1)) * R + prow) * P + u0 + (warp & 1) * 8 + chunk);
            send4(at_rank(dst, (uint32_t)peer), at_rank(next_bar, (uint32_t)peer), v);
          }
        }
        cs[i * THREADS + tid] = c;
        if (i + 1 == tiles) xp += step_x;
        const int ni = i + 1 < tiles ? i + 1 : 0;
        if ((ni > 0 || p + 1 < T) && row_begin + ni * R + prow < row_end && unit_ok) x = xp[ni * tile_x];
        if (mine) {
          if (gp != nullptr) gp[(long long)i * R * 4 * U] = act;
          if (sp != nullptr && (gate != 0 || p + 1 < T)) sp[i * tile_s] = gate == 1 ? c : h;
          if (gate == 3 && p + 1 == T) {
            const size_t at = (size_t)(row_begin + i * R + prow) * U + u0 + pu;
            a.hT[at] = h;
            a.cT[at] = c;
          }
        }
      }
    }
    if (gp != nullptr) gp += 4 * step_c;
    if (sp != nullptr) sp += step_s;
  }
  if (!ok && tid == 0) atomicExch(a.err, 42);
  cluster_meet();  // a peer that is late still writes here
}

template <int R>
__global__ void __launch_bounds__(cluster_threads<R>(), 1) lstm_cluster_backward_kernel(const LstmArgs a) {
  constexpr int RP = padded_rows(R), PART = peer_part(R), RC = row_chunk<R>();
  extern __shared__ float4 smem4[];
  __shared__ alignas(8) unsigned long long bars[TILES_MAX * 2];
  const int U = a.U, T = a.T, B = a.B, S = a.slices, K = 4 * U;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x % S, group = blockIdx.x / S;
  const int u0 = slice * UNITS, nu = min(UNITS, U - u0);
  const int row_begin = group * a.rows_per_group, row_end = min(B, row_begin + a.rows_per_group);
  const int tiles = (row_end - row_begin + R - 1) / R;
  float* recv = reinterpret_cast<float*>(smem4);                      // [tile][2][S][PART]
  float* dzs = recv + (size_t)(a.rows_per_group / R) * 2 * S * PART;  // [2][R][DZ_ROW]: gate gradients of this CTA's units
  float* dcs = dzs + 2 * R * DZ_ROW;                                  // [tile][16 R]: the running gradient of c
  const uint32_t bytes = (uint32_t)(S * UNITS * RP * 4);
  if (tid == 0) {
    for (int i = 0; i < tiles * 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_u32(bars + i)));
      expect(shared_u32(bars + i), bytes);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Products: warp w has the 16 units of peer w, a lane two of them and the 16 columns of one gate.
  const int kq = lane & 3, uw = (lane >> 2) * 2;
  unsigned long long w[2][UNITS / 2];
  if (warp < S) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < UNITS; k += 2) {
        const int u = warp * UNITS + uw + j;
        const float* src = a.R + (size_t)u * K + (size_t)kq * U + u0 + k;
        w[j][k / 2] = pair_of(u < U && k < nu ? src[0] : 0.f, u < U && k + 1 < nu ? src[1] : 0.f);
      }
  }
  // Pointwise part: four lanes, one a gate, for each (unit, row)
  const int cell = warp * 8 + (lane & 7), gate = lane >> 3, l8 = lane & 7;
  const bool pointwise = warp < 2 * R;
  const int pu = pointwise ? cell / R : 0, prow = pointwise ? cell % R : 0;
  const bool active = pointwise && pu < nu;
  const int last = a.dh0 != nullptr ? -1 : 0;  // step -1 only carries the gradient on to h0
  const size_t first = (size_t)(row_begin + prow);
  const long long step_z = a.reverse ? -(long long)K : (long long)K, step_c = (long long)B * U;
  float* zp = a.dz + (first * T + (a.reverse ? 0 : T - 1)) * K + (size_t)gate * U + u0 + pu;  // of the present step, tile 0
  // The next item's values, a step ahead of their use: this lane's gate, and one of c, the c before and the gradient of the output
  const float* gp = a.gates + (first + (size_t)(T - 1) * B) * K + (size_t)gate * U + u0 + pu;
  const float* ap = gate == 0 ? a.cs + (first + (size_t)(T - 1) * B) * U + u0 + pu
                  : gate == 1 ? (T > 1 ? a.cs + (first + (size_t)(T - 2) * B) * U + u0 + pu : a.c0 + first * U + u0 + pu)
                  : gate == 2 && a.dout != nullptr ? a.dout + (first * T + T - 1) * U + u0 + pu : nullptr;
  const long long step_a = gate == 2 ? U : step_c, tile_a = gate == 2 ? (long long)R * T * U : (long long)R * U;
  float gv = 0.f, aux = 0.f;
  auto fetch = [&](int q, int i) {  // gp and ap stand at step q
    if (q < 0 || !active || row_begin + i * R + prow >= row_end) return;
    gv = gp[(long long)i * R * K];
    if (ap != nullptr) aux = ap[i * tile_a];
  };
  fetch(T - 1, 0);
  cluster_meet();

  bool ok = true;
  int item = 0;
  for (int q = T - 1; q >= last && ok; --q) {
    const int s = T - 1 - q, b = s & 1;
    for (int i = 0; i < tiles; ++i, ++item) {
      const uint32_t bar = shared_u32(bars + i * 2 + b), next_bar = shared_u32(bars + i * 2 + (b ^ 1));
      float* dz = dzs + (item & 1) * R * DZ_ROW;  // two: slower warps still multiply the one before
      if (pointwise) {
        const bool mine = active && row_begin + i * R + prow < row_end;
        const size_t at = (first + i * R) * U + u0 + pu;
        // what does not depend on the peers
        const float gi = __shfl_sync(0xffffffffu, gv, l8), gf = __shfl_sync(0xffffffffu, gv, 8 + l8);
        const float gg = __shfl_sync(0xffffffffu, gv, 16 + l8), go = __shfl_sync(0xffffffffu, gv, 24 + l8);
        const float c = __shfl_sync(0xffffffffu, aux, l8), c_before = __shfl_sync(0xffffffffu, aux, 8 + l8), dy = __shfl_sync(0xffffffffu, aux, 16 + l8);
        const float tc = tanhf(c), through = go * (1.f - tc * tc);
        const float slope = gate == 0 ? gg * gi * (1.f - gi) : gate == 1 ? c_before * gf * (1.f - gf) : gate == 2 ? gi * (1.f - gg * gg) : tc * go * (1.f - go);
        float dh = q >= 0 ? dy : 0.f, dc = 0.f;
        if (s == 0) {
          if (mine && a.dhT != nullptr) dh += a.dhT[at];
          if (mine && a.dcT != nullptr) dc = a.dcT[at];
        } else {
          dc = dcs[i * UNITS * R + cell];
          ok = received(bar, (uint32_t)((s - 1) >> 1) & 1u);
          const float* r = recv + (size_t)(i * 2 + b) * S * PART + pu * RP + prow;
          float sum = 0.f;
          for (int v = gate; v < S; v += 4) sum += r[v * PART];
          sum += __shfl_xor_sync(0xffffffffu, sum, 8);
          sum += __shfl_xor_sync(0xffffffffu, sum, 16);
          dh += sum;
        }
        float d = 0.f;
        if (mine && q >= 0) {
          dc += dh * through;
          d = (gate == 3 ? dh : dc) * slope;
        }
        dz[prow * DZ_ROW + gate * DZ_GATE + pu] = d;
        __syncwarp();  // the four lanes have read dcs
        if (gate == 0) dcs[i * UNITS * R + cell] = dc * gf;
        if (mine && q >= 0) {
          zp[(long long)i * R * T * K] = d;
          if (q == 0 && gate == 0) a.dc0[at] = dc * gf;
        }
        if (mine && q < 0 && gate == 0) a.dh0[at] = dh;
        if (i + 1 == tiles) {
          gp -= 4 * step_c;
          if (gate == 1 && q == 1) ap = a.c0 + first * U + u0 + pu;  // step 0 follows: the c before it
          else if (ap != nullptr) ap -= step_a;
          zp -= step_z;
        }
        fetch(i + 1 < tiles ? q : q - 1, i + 1 < tiles ? i + 1 : 0);
      }
      ok = __syncthreads_and(ok);
      if (!ok) break;
      if (tid == 0 && s > 0 && q - 2 >= last) expect(bar, bytes);
      if (q > last && warp < S) {
        float v[RP];
#pragma unroll
        for (int r = R; r < RP; ++r) v[r] = 0.f;
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += RC) {
          unsigned long long acc[RC][2];
#pragma unroll
          for (int r = 0; r < RC; ++r) acc[r][0] = acc[r][1] = 0ull;
#pragma unroll
          for (int k = 0; k < UNITS / 4; ++k) {
#pragma unroll
            for (int r = 0; r < RC; ++r) {
              const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(dz + (r0 + r) * DZ_ROW + kq * DZ_GATE + k * 4);
              acc[r][0] = fma2(d.x, w[0][2 * k], acc[r][0]);
              acc[r][1] = fma2(d.x, w[1][2 * k], acc[r][1]);
              acc[r][0] = fma2(d.y, w[0][2 * k + 1], acc[r][0]);
              acc[r][1] = fma2(d.y, w[1][2 * k + 1], acc[r][1]);
            }
          }
          // the four gates' sums: a pair of lanes swaps units, after which two pairs have the same two
#pragma unroll
          for (int r = 0; r < RC; ++r) {
            const float e0 = sum_of(acc[r][0]), e1 = sum_of(acc[r][1]);
            const float one = (kq & 1 ? e1 : e0) + __shfl_xor_sync(0xffffffffu, kq & 1 ? e0 : e1, 1);
            v[r0 + r] = one + __shfl_xor_sync(0xffffffffu, one, 2);
          }
        }
        const uint32_t dst = at_rank(shared_u32(recv + ((size_t)(i * 2 + (b ^ 1)) * S + slice) * PART + (uw + (kq & 1)) * RP), (uint32_t)warp);
        const uint32_t peer_bar = at_rank(next_bar, (uint32_t)warp);
#pragma unroll
        for (int r = 0; r < RP; r += 4)
          if ((r / 4 & 1) == kq >> 1) send4(dst + r * 4, peer_bar, make_float4(v[r], v[r + 1], v[r + 2], v[r + 3]));
      }
    }
  }
  if (!ok && tid == 0) atomicExch(a.err, 43);
  cluster_meet();
}

typedef void (*LstmKernel)(const LstmArgs);
struct ClusterPlan {
  int rows = 0, tiles = 0;  // rows of a tile, tiles of a cluster; 0: not on clusters
  LstmKernel forward = nullptr, backward = nullptr;
  int threads = 0;
  size_t smem_forward = 0, smem_backward = 0;
};

template <int R>
bool allow_plan(const ClusterPlan& c, int U);

// false: the device refuses a kernel
template <int R>
bool fill_plan(ClusterPlan& c, int S, int U) {
  const int kw = U <= 64 ? 4 : U <= 128 ? 8 : U <= 192 ? 12 : 16;
  c.rows = R;
  c.threads = cluster_threads<R>();
  c.forward = kw == 4 ? lstm_cluster_forward_kernel<R, 4> : kw == 8 ? lstm_cluster_forward_kernel<R, 8> : kw == 12 ? lstm_cluster_forward_kernel<R, 12>
                                                                                                       : lstm_cluster_forward_kernel<R, 16>;
  c.backward = lstm_cluster_backward_kernel<R>;
  c.smem_forward = ((size_t)c.tiles * 2 * R * GEMV_WARPS * kw + 2 * GEMV_WARPS * R * COLS + (size_t)c.tiles * c.threads) * 4;
  c.smem_backward = ((size_t)c.tiles * 2 * S * peer_part(R) + 2 * R * DZ_ROW + (size_t)c.tiles * UNITS * R) * 4;
  return allow_plan<R>(c, U);
}
constexpr int CLUSTER_SMEM = 200 * 1024;  // above the largest of these: four tiles of ten rows, 256 units forward 174 KB, backward 110

bool allow(LstmKernel k) {
  const bool fine = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CLUSTER_SMEM) == cudaSuccess &&
                    cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (!fine) cudaGetLastError();
  return fine;
}
// The kernels of a plan, asked for once per device: each one that is named is loaded, so none that the size does not take.
template <int R>
bool allow_plan(const ClusterPlan& c, int U) {
  static signed char known[KB_MAX_DEVICES][4] = {{0}};  // by the K width; 0: not asked, 1: fine, -1: refused
  signed char& slot = known[kb_device_slot()][U <= 64 ? 0 : U <= 128 ? 1 : U <= 192 ? 2 : 3];
  if (slot == 0) slot = allow(c.forward) && allow(c.backward) ? 1 : -1;
  return slot > 0;
}

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int S) {
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

// Clusters of `S` CTAs, one an SM, that run at once (a GPC has to hold a whole one: 7 of sixteen CTAs, 15 of eight, 33 of four on a B200), or
// 0 where the kernel is refused.  Asked once per device and size.
int active_clusters(int S) {
  static int known[KB_MAX_DEVICES][CLUSTER_MAX + 1] = {{0}};  // 0: not asked; else 1 + answer
  int& slot = known[kb_device_slot()][S];
  if (slot == 0) {
    int n = 0;
    bool fine = allow(lstm_cluster_forward_kernel<10, 16>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S * 64);
    cfg.blockDim = dim3(cluster_threads<10>());
    cfg.dynamicSmemBytes = CLUSTER_SMEM;
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, S);
    fine = fine && cudaOccupancyMaxActiveClusters(&n, (LstmKernel)lstm_cluster_forward_kernel<10, 16>, &cfg) == cudaSuccess;
    if (!fine) cudaGetLastError();
    slot = 1 + (fine ? n : 0);
  }
  return slot - 1;
}

// The smallest tiles whose clusters hold all rows at once, up to four of ten rows a cluster, and in as many even waves as it takes beyond that: four full
// tiles in each wave but the last leave that one half empty (1024 rows x 96 units, 20 steps: forward 294 us, even 184; the kernels above 257).
// Clusters of eleven or twelve CTAs hold half of the SMs, one a GPC.  From the second wave on, a forward step of the kernels above, which hold all,
// is then the shorter one where it has fewer than 10 / 17 of the rows one after the other (512 rows x 176 units: 80 rows 349 us, 40 rows 298; 1024 x 192:
// 707 and 721); backward, what they send through L2 keeps them behind (866 and 942).
ClusterPlan cluster_plan(int B, int U, bool backward) {
  ClusterPlan c;
  if (B <= 0 || U <= 0 || U % 4 || U > CLUSTER_UNITS) return c;
  const int S = (U + UNITS - 1) / UNITS, at_once = active_clusters(S);
  if (at_once <= 0) return c;
  const int waves = (B + at_once * 10 * TILES_MAX - 1) / (at_once * 10 * TILES_MAX);
  const int each = (B + at_once * waves - 1) / (at_once * waves);  // rows of a cluster
  c.tiles = (each + 9) / 10;
  if (!backward && waves > 1 && S > 10 && S <= 12) {
    const int groups = kb_sm_count() / S, tiles = (B + ROWS - 1) / ROWS;
    if (waves * c.tiles * 10 * 10 > (tiles + groups - 1) / groups * ROWS * 17) return ClusterPlan{};
  }
  const int rows = (each + c.tiles - 1) / c.tiles;
  const bool fine = rows <= 2 ? fill_plan<2>(c, S, U) : rows <= 4 ? fill_plan<4>(c, S, U) : rows <= 8 ? fill_plan<8>(c, S, U) : fill_plan<10>(c, S, U);
  return fine ? c : ClusterPlan{};
}

size_t lstm_smem(int U, bool backward) {
  const size_t r = (size_t)U * COLS * 4;
  return backward ? r + ROWS * (KC + 4) * 4 + 32 * ROWS * UNITS * 4 : r + ROWS * (U + 4) * 4 + WARPS * ROWS * COLS * 4;
}
}  // namespace

// Whether this direction of the layer runs on clusters, which need no counters.
KB_API int kb200_lstm_clustered(int B, int U, int backward) { return cluster_plan(B, U, backward != 0).rows > 0 ? 1 : 0; }

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
  const ClusterPlan plan = cluster_plan(B, U, backward != 0);
  if (plan.rows > 0) {
    a.rows_per_group = plan.rows * plan.tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.slices * ((B + a.rows_per_group - 1) / a.rows_per_group)));
    cfg.blockDim = dim3((unsigned)plan.threads);
    cfg.dynamicSmemBytes = backward ? plan.smem_backward : plan.smem_forward;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    cluster_config(cfg, at, a.slices);
    if (cudaLaunchKernelEx(&cfg, backward ? plan.backward : plan.forward, a) != cudaSuccess) {
      kb200_set_error(cudaGetErrorString(cudaGetLastError()));
      return -1;
    }
    return 0;
  }
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
