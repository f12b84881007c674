// Products of few rows with weights as they are stored: C[M, N] = act(A[M, K] x W[K, N] + bias), M <= 128, W float32 or bf16, tcgen05.
//
// Inference on a handful of tokens reads every weight once and does little else: the bound is the weights' bytes.  A float32 weight used
// to be read, written as bf16 by a cast of its own and read again by the library's product; here its tiles go through registers,
// where they are rounded, straight into the swizzled operand layout in shared memory, and no copy of the weight exists.  A CTA has 64
// columns and walks the whole of K, three CTAs an SM with some 48 KB of weights in flight, so it takes a weight of many columns: a
// vocabulary.  CTAs that share K would have narrower ones run as quickly, but their sums round otherwise than those of the layers' own calls,
// which run along K, and a first call would differ from a second one.
//
// Every wait is bounded: on expiry the kernel records a code in *err and returns.
#include "gemm_sm100.cuh"

namespace {
using namespace kbgemm;

namespace rw {
constexpr int BM = 128, BN = 64, BK = 64, STAGES = 3;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE = A_BYTES + B_BYTES;
constexpr int LOADERS = 128, THREADS = LOADERS + 64;  // warps 0-3: weights, then the epilogue; 4: copies of A; 5: MMA
constexpr int SUM_PITCH = BN + 4;                     // floats a row of the sums: 16-byte accesses of neighbouring rows hit different banks
constexpr int SMEM = STAGES * STAGE + 1024 + 128;
static_assert(BM * SUM_PITCH * 4 <= STAGES * STAGE, "the sums reuse the operand stages");
constexpr uint32_t LIMIT = 1u << 20;
}  // namespace rw

constexpr int MAX_WEIGHTS = 3;
struct RowsParams {
  const void* w[MAX_WEIGHTS];     // weights side by side (the three projections of an attention layer): columns [start, start + width) of C
  const void* bias[MAX_WEIGHTS];
  int start[MAX_WEIGHTS], width[MAX_WEIGHTS];
  int vec[MAX_WEIGHTS];           // rows of this weight start on 16-byte lines
  int weights;
  void* out;
  int M, K;
  long long ldo;
  int act, bias16, apart;
  int* err;
};
struct WView {  // the weight of a tile
  const void* w;
  int N, n0, K, vec;  // its width (and row pitch), the tile's first column in it
};

__device__ __forceinline__ bool rows_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t it = 0; it < rw::LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort_flag) return false;
  }
  return false;
}

// One K block of W as bf16: chunk c of a thread is 8 columns of one row (row-major over 64 rows x 8 chunks).
template <typename T>
struct WTile {
  uint4 v[4];
  __device__ __forceinline__ void load(const WView& p, int k0, int tid) {
    const int n0 = p.n0;
    if (p.vec) {
      float4 lo[4], hi[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = c * rw::LOADERS + tid, k = k0 + (i >> 3), n = n0 + (i & 7) * 8;
        if constexpr (sizeof(T) == 4) {
          const float* s = reinterpret_cast<const float*>(p.w) + (size_t)k * p.N + n;
          lo[c] = k < p.K && n < p.N ? *reinterpret_cast<const float4*>(s) : make_float4(0.f, 0.f, 0.f, 0.f);
          hi[c] = k < p.K && n + 4 < p.N ? *reinterpret_cast<const float4*>(s + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
          const __nv_bfloat16* s = reinterpret_cast<const __nv_bfloat16*>(p.w) + (size_t)k * p.N + n;
          v[c] = k < p.K && n < p.N ? *reinterpret_cast<const uint4*>(s) : make_uint4(0, 0, 0, 0);
        }
      }
      if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float f[8] = {lo[c].x, lo[c].y, lo[c].z, lo[c].w, hi[c].x, hi[c].y, hi[c].z, hi[c].w};
          const bf16x8 pk = pack8(f);
          v[c] = *reinterpret_cast<const uint4*>(&pk);
        }
      }
    } else {
      // rows that start anywhere: 32 columns of a row an instruction.  Element j of a thread is row j of a group of sixteen, column
      // `lane` or `lane + 32`; two bf16 share a register
      uint32_t* u = reinterpret_cast<uint32_t*>(v);
      const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int k = k0 + warp * 16 + j;
        const T* s = reinterpret_cast<const T*>(p.w) + (size_t)k * p.N + n0 + lane;
        const T a = k < p.K && n0 + lane < p.N ? s[0] : from_f32<T>(0.f), b = k < p.K && n0 + lane + 32 < p.N ? s[32] : from_f32<T>(0.f);
        const __nv_bfloat162 h = __floats2bfloat162_rn(to_f32<T>(a), to_f32<T>(b));
        u[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
  }
  // MN-major operand: one row of 128 bytes a K index, its eight 16-byte chunks swizzled by the row
  __device__ __forceinline__ void store(uint32_t dst, int vec, int tid) const {
    if (vec) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = c * rw::LOADERS + tid, k = i >> 3, n = i & 7;
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (uint32_t)(k * 128 + ((n ^ (k & 7)) << 4))), "r"(v[c].x), "r"(v[c].y), "r"(v[c].z),
                     "r"(v[c].w) : "memory");
      }
    } else {
      const uint32_t* u = reinterpret_cast<const uint32_t*>(v);
      const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int k = warp * 16 + j;
        const uint32_t row = dst + (uint32_t)(k * 128 + (lane & 7) * 2);
        asm volatile("st.shared.b16 [%0], %1;" ::"r"(row + (uint32_t)((((lane >> 3)) ^ (k & 7)) << 4)), "h"((uint16_t)(u[j] & 0xffffu)) : "memory");
        asm volatile("st.shared.b16 [%0], %1;" ::"r"(row + (uint32_t)((((lane >> 3) + 4) ^ (k & 7)) << 4)), "h"((uint16_t)(u[j] >> 16)) : "memory");
      }
    }
  }
};

template <typename T>
__global__ void __launch_bounds__(rw::THREADS, 3) gemm_rows_kernel(const __grid_constant__ CUtensorMap map_a, const RowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + rw::STAGES * rw::STAGE;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (rw::STAGES + s); };
  const uint32_t done = bars + 8u * (2 * rw::STAGES);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + rw::STAGES * rw::STAGE + 8 * (2 * rw::STAGES + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * rw::BN;
  const int which = p.weights > 2 && n0 >= p.start[2] ? 2 : p.weights > 1 && n0 >= p.start[1] ? 1 : 0;
  const WView wv{p.w[which], p.width[which], n0 - p.start[which], p.K, p.vec[which]};
  const int blocks = (p.K + rw::BK - 1) / rw::BK;

  if (tid == rw::LOADERS) {
    prefetch_map(&map_a);
    for (int s = 0; s < rw::STAGES; ++s) {
      mbar_init(full(s), 1 + rw::LOADERS / 32);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(smem_u32((const void*)tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 4) {
    if (elect_one()) {
      bool ok = true;
      int issued = 0;
      for (int b = 0; b < blocks && ok; ++b) {
        const int s = b % rw::STAGES;
        ok = rows_wait(empty(s), ((b / rw::STAGES) & 1) ^ 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(full(s), rw::A_BYTES);
        tma_load_2d(base + s * rw::STAGE, &map_a, full(s), b * rw::BK, 0);
        issued = b + 1;
      }
      if (!ok) {
        if (p.err) atomicExch(p.err, 51);
        *abort_flag = 1;
        for (int i = 0; i < 1024 && issued > 0; ++i) __nanosleep(1000);  // about a millisecond for the copies in flight
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      // fp32 accumulate, bf16 operands, A K-major, W MN-major
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(rw::BN >> 3) << 17) | ((uint32_t)(rw::BM >> 4) << 24);
      bool ok = true;
      for (int b = 0; b < blocks; ++b) {
        const int s = b % rw::STAGES;
        ok = rows_wait(full(s), (b / rw::STAGES) & 1, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t adesc = make_smem_desc(base + s * rw::STAGE, false), bdesc = make_smem_desc(base + s * rw::STAGE + rw::A_BYTES, true);
#pragma unroll
        for (int k = 0; k < rw::BK / UMMA_K; ++k)
          umma_bf16(tmem, adesc + (uint64_t)((32u >> 4) * k), bdesc + (uint64_t)((2048u >> 4) * k), idesc, (b > 0 || k > 0) ? 1u : 0u);
        umma_commit(empty(s));
      }
      if (ok) {
        umma_commit(done);
      } else {
        if (p.err) atomicExch(p.err, 52);
        *abort_flag = 1;
      }
    }
  } else {
    bool ok = true;
    WTile<T> tile;
    tile.load(wv, 0, tid);
    for (int b = 0; b < blocks && ok; ++b) {
      const int s = b % rw::STAGES;
      WTile<T> next;
      if (b + 1 < blocks) next.load(wv, (b + 1) * rw::BK, tid);
      ok = rows_wait(empty(s), ((b / rw::STAGES) & 1) ^ 1, abort_flag);
      if (!ok) break;
      tile.store(base + s * rw::STAGE + rw::A_BYTES, wv.vec, tid);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads what these threads wrote
      __syncwarp();
      if (lane == 0) mbar_arrive(full(s));
      tile = next;
    }
    ok = ok && rows_wait(done, 0, abort_flag);
    if (ok) {
      // every MMA has read its operands: the stages now hold this CTA's sums, rows of SUM_PITCH floats
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t r[64];
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), r);
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + 32, r + 32);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      float* row = reinterpret_cast<float*>(base_ptr) + (size_t)tid * rw::SUM_PITCH;
#pragma unroll
      for (int j = 0; j < 64; j += 4)
        *reinterpret_cast<float4*>(row + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
    } else {
      if (lane == 0 && p.err) atomicExch(p.err, 53);
      *abort_flag = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(tmem) : "memory");
  // Rows of the result, eight columns a thread
  const void* bias = p.bias[which];
  const int width = min(rw::BN, (int)p.ldo - n0);  // columns of the output's rows, their padding included
  for (int i = tid; i < p.M * 8; i += rw::THREADS) {
    const int row = i >> 3, c = (i & 7) * 8;
    if (c >= width) continue;
    const float* sum = reinterpret_cast<const float*>(base_ptr) + (size_t)row * rw::SUM_PITCH + c;
    const float4 lo = *reinterpret_cast<const float4*>(sum), hi = *reinterpret_cast<const float4*>(sum + 4);
    float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = wv.n0 + c + j;
      if (p.apart) v[j] = __bfloat162float(__float2bfloat16(v[j]));
      if (bias != nullptr && n < wv.N)  // in the layer's type, as the layer itself reads it
        v[j] += __bfloat162float(p.bias16 ? reinterpret_cast<const __nv_bfloat16*>(bias)[n] : __float2bfloat16(reinterpret_cast<const float*>(bias)[n]));
      v[j] = apply_act<false>(v[j], p.act);
    }
    const bf16x8 pk = pack8(v);
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)row * p.ldo + n0 + c) = *reinterpret_cast<const uint4*>(&pk);
  }
}

template <typename T>
int launch_rows(const CUtensorMap& map_a, const RowsParams& p, int n_tiles, cudaStream_t stream) {
  static bool attr[KB_MAX_DEVICES] = {false};
  if (!kb_allow_smem(gemm_rows_kernel<T>, rw::SMEM, attr)) {
    kb200_set_error("gemm_rows: cannot raise the shared-memory limit of the kernel on this device");
    return -3;
  }
  gemm_rows_kernel<T><<<(unsigned)n_tiles, rw::THREADS, rw::SMEM, stream>>>(map_a, p);
  KB_CHECK_LAUNCH("gemm_rows");
  return 0;
}

// Weights for the GEMM of many rows: W_i [K, N_i] float32 or bf16 of any width into columns [start, start + 8 vecs) of a bf16 matrix, zeros
// behind N_i, and their biases rounded to bf16 beside it.  Bound by its traffic: [768, 50257] float32, 231 MB: 44 us; a cast and a padding
// pass of its own took 24 + 31.
struct PlaceParams {
  const void* w[MAX_WEIGHTS];
  const float* bias[MAX_WEIGHTS];
  int start[MAX_WEIGHTS], width[MAX_WEIGHTS], vecs[MAX_WEIGHTS];
  long long end[MAX_WEIGHTS];  // blocks up to the end of this weight
  int vec[MAX_WEIGHTS];
  int rows;
  __nv_bfloat16* dst;
  float* bias_out;
  long long ldd;
};
template <typename T>
__global__ void __launch_bounds__(256) place_weight_kernel(const PlaceParams p) {
  const int which = blockIdx.x < p.end[0] ? 0 : blockIdx.x < p.end[1] ? 1 : 2;
  const int N = p.width[which], vecs = p.vecs[which];
  const long long i = ((long long)blockIdx.x - (which > 0 ? p.end[which - 1] : 0)) * 256 + threadIdx.x;
  if (p.bias_out != nullptr && i < vecs) {
    const float* bias = p.bias[which];
    float* to = p.bias_out + p.start[which] + i * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) to[j] = bias != nullptr && i * 8 + j < N ? __bfloat162float(__float2bfloat16(bias[i * 8 + j])) : 0.f;
  }
  const long long r = i / vecs;
  if (r >= p.rows) return;
  const int v = (int)(i - r * vecs);
  const T* s = reinterpret_cast<const T*>(p.w[which]) + r * N + (long long)v * 8;
  float f[8];
  if (p.vec[which] && sizeof(T) == 4 && v * 8 < N) {
    const float4 lo = *reinterpret_cast<const float4*>(s), hi = v * 8 + 4 < N ? *reinterpret_cast<const float4*>(s + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    f[0] = lo.x, f[1] = lo.y, f[2] = lo.z, f[3] = lo.w, f[4] = hi.x, f[5] = hi.y, f[6] = hi.z, f[7] = hi.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = v * 8 + j < N ? to_f32<T>(s[j]) : 0.f;
  }
  const bf16x8 pk = pack8(f);
  *reinterpret_cast<uint4*>(p.dst + r * p.ldd + p.start[which] + (long long)v * 8) = *reinterpret_cast<const uint4*>(&pk);
}

// Up to three weights side by side and their biases behind one another; false: too large for a launch.
bool place(const void* const* w, const void* const* b, const int* n, int count, __nv_bfloat16* matrix, float* bias, int K, long long ld, int w_fp32, cudaStream_t stream) {
  PlaceParams p{};
  long long blocks = 0;
  for (int i = 0, at = 0; i < MAX_WEIGHTS; at += n[i], ++i) {
    if (i < count) {
      p.w[i] = w[i], p.bias[i] = (const float*)b[i], p.start[i] = at, p.width[i] = n[i];
      p.vecs[i] = count == 1 ? (int)(ld / 8) : (n[i] + 7) / 8;
      p.vec[i] = ((uintptr_t)w[i] & 15) == 0 && n[i] % 4 == 0;
      blocks += ((long long)K * p.vecs[i] + 255) / 256;
    }
    p.end[i] = blocks;
  }
  if (blocks > 0x7fffffffll) return false;
  p.rows = K, p.dst = matrix, p.bias_out = bias, p.ldd = ld;
  if (w_fp32) place_weight_kernel<float><<<(unsigned)blocks, 256, 0, stream>>>(p);
  else place_weight_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, stream>>>(p);
  return true;
}

// out = relu?(out + bias) on contiguous bf16 rows of `ld` columns, a multiple of 8; the bias in bf16 or float32, its first `n` columns
__global__ void __launch_bounds__(256) bias_rows_kernel(uint4* __restrict__ out, const void* __restrict__ bias, long long vecs, int per_row, int n, int bias16, int relu) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= vecs) return;
  const int c = (int)(i % per_row) * 8;
  const uint4 raw = out[i];
  const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&raw);
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = __bfloat162float(h[j]);
    if (bias != nullptr && c + j < n) v[j] += bias16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[c + j]) : reinterpret_cast<const float*>(bias)[c + j];
    if (relu) v[j] = v[j] <= 0.f ? 0.f : v[j];  // a NaN stays one
  }
  const bf16x8 pk = pack8(v);
  out[i] = *reinterpret_cast<const uint4*>(&pk);
}
}  // namespace

KB_API int kb200_gemm_bf16_run(const void* a, const void* b, void* c, const void* bias, int M, int N, int K, long long lda, long long ldb, long long ldc,
                               int a_mn_major, int b_mn_major, int act, int out_fp32, int bias_bf16, int split_k, int variant, int* err, cudaStream_t stream);

// C[M, ldo] (bf16, contiguous rows) = act(A x [W0 W1 W2] + bias): A bf16 [M, K], pitch lda; W_i [K, n_i] contiguous, all float32 (w_fp32) or
// bf16; biases per weight, float32 (rounded to bf16 as they are read) or (bias16) bf16, null where there is none.  More than one weight:
// widths that are multiples of 64.  ldo: the sum of the widths up to the next multiple of 8, or of 64 for one odd width; the columns behind it
// hold act(0).
// rows: by the kernel for few rows (M <= 128), which needs no scratch.  apart: the product is rounded before the bias, as two operations would
// leave it (act: none or relu).  scratch: a bf16 matrix [K, ldo] and ldo floats behind it, or null if
// there is one bf16 weight whose width is a multiple of 8, without a bias in float32.
KB_API int kb200_dense_infer(const void* a, const void* w0, const void* w1, const void* w2, const void* b0, const void* b1, const void* b2, int n0, int n1, int n2,
                             void* out, void* scratch, int M, int K, long long lda, long long ldo, int w_fp32, int bias16, int act, int rows, int apart, int* err,
                             cudaStream_t stream) {
  if (M <= 0 || K <= 0 || n0 <= 0) return 0;
  const void* w[MAX_WEIGHTS] = {w0, w1, w2};
  const void* b[MAX_WEIGHTS] = {b0, b1, b2};
  const int n[MAX_WEIGHTS] = {n0, n1, n2};
  const int count = n2 > 0 ? 3 : n1 > 0 ? 2 : 1, total = n0 + n1 + n2;
  const bool has_bias = b0 != nullptr || b1 != nullptr || b2 != nullptr;
  // one odd width in whole 128-byte lines (a matrix of its own then)
  const bool wider = !rows && count == 1 && n0 % 8 && ldo == (total + 63ll) / 64 * 64;
  if ((lda % 8) || (K % 8) || (rows && M > rw::BM) || (apart && act != ACT_NONE && act != ACT_RELU) || !(ldo == (total + 7) / 8 * 8 || wider) || (((uintptr_t)a | (uintptr_t)out | (uintptr_t)scratch) & 15) ||
      (count > 1 && ((n0 % 64) || (n1 % 64) || (n2 % 64) || bias16)) || (bias16 && n0 % 8)) {
    kb200_set_error("dense_infer: 16-byte aligned operands, pitches in multiples of 8, several weights only in multiples of 64 columns with float32 biases, odd widths with float32 ones");
    return -2;
  }
  if (rows) {
    CUtensorMap map_a;
    if (!make_map(&map_a, a, K, M, lda, rw::BK, rw::BM)) {
      kb200_set_error("dense_infer: cuTensorMapEncodeTiled failed");
      return -3;
    }
    RowsParams p{};
    for (int i = 0, at = 0; i < count; at += n[i], ++i) {
      p.w[i] = w[i], p.bias[i] = b[i], p.start[i] = at, p.width[i] = n[i];
      p.vec[i] = ((uintptr_t)w[i] & 15) == 0 && n[i] % (w_fp32 ? 4 : 8) == 0;
    }
    p.weights = count, p.out = out, p.M = M, p.K = K, p.ldo = ldo, p.act = act, p.bias16 = bias16, p.apart = apart, p.err = err;
    const int n_tiles = (total + rw::BN - 1) / rw::BN;
    return w_fp32 ? launch_rows<float>(map_a, p, n_tiles, stream) : launch_rows<__nv_bfloat16>(map_a, p, n_tiles, stream);
  }
  const __nv_bfloat16* matrix = (const __nv_bfloat16*)w0;
  const void* bias = b0;
  if (scratch != nullptr) {
    __nv_bfloat16* to = (__nv_bfloat16*)scratch;
    float* placed = has_bias && !bias16 ? (float*)(to + (size_t)K * ldo) : nullptr;
    if (!place(w, b, n, count, to, placed, K, ldo, w_fp32, stream)) {
      kb200_set_error("dense_infer: weight too large for one launch");
      return -2;
    }
    KB_CHECK_LAUNCH("place_weight");
    matrix = to, bias = bias16 ? b0 : placed;
  } else if (w_fp32 || count > 1 || n0 % 8 || (has_bias && !bias16)) {
    kb200_set_error("dense_infer: these weights need a scratch matrix");
    return -2;
  }
  const int rc = kb200_gemm_bf16_run(a, matrix, out, apart ? nullptr : bias, M, (int)ldo, K, lda, ldo, ldo, 0, 1, apart ? ACT_NONE : act, 0, bias16, 1, 0, err, stream);
  if (rc != 0 || !apart || (!has_bias && act == ACT_NONE)) return rc;
  const long long vecs = (long long)M * (ldo / 8);
  if (vecs / 256 > 0x7ffffff0ll) {
    kb200_set_error("dense_infer: result too large for one launch");
    return -2;
  }
  bias_rows_kernel<<<(unsigned)((vecs + 255) / 256), 256, 0, stream>>>((uint4*)out, has_bias ? bias : nullptr, vecs, (int)(ldo / 8), total, bias16, act == ACT_RELU);
  KB_CHECK_LAUNCH("bias_rows");
  return 0;
}
