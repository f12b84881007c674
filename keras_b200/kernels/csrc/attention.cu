// Flash attention forward on tcgen05 tensor cores: O = softmax(scale * Q K^T [+ mask]) V without materialising the score matrix.
// Layout [batch, time, heads, head_dim] for Q, K, V and O (the layout of the attention layers), bf16 in and out, fp32
// statistics; grouped-query attention by mapping query head h to key/value head h / (H / Hkv).
// Replaces the einsum -> masked softmax -> einsum chain (keras/src/layers/attention/multi_head_attention.py:574-608) and the
// library call behind keras/src/backend/torch/nn.py:1124-1175.
//
// One CTA per (NT x 128 query rows, head, batch element):
//   softmax warps  four per tile of 128 rows, one thread per query row (= TMEM lane): the row of S in registers, maximum and sum
//                  without any shuffle, P (bf16) written back over S in TMEM
//   TMA warp       Q once, then K and V blocks of 128 keys through one ring (4-D tiled copies, 128-byte swizzle)
//   MMA warp       one elected thread: S = Q K^T into TMEM, O += P V with P as the TMEM operand and O accumulated in TMEM
// With two tiles (NT = 2, one CTA per SM) the tensor pipe works for one tile while the other tile's softmax runs.  Products run
// in issue order, so the score product of block j + 1 may follow P V of block j on the same TMEM columns, and a full S also says
// that the previous P V is done.  O is rescaled only when a row's maximum has grown by more than 2^8 since the last time (its P
// would otherwise leave the range that bf16 and the fp32 sums hold comfortably); the final division by the sum makes up for the
// rest exactly.  Prompts of at most 128 rows take NT = 1 and two CTAs per SM.
// What bounds it: at head size 64 the exponentials (16 a cycle and SM: 1024 cycles a tile and block, a quarter of them moved to
// the FMA pipe) and the latency from S over P to the next S; at 128 the tensor pipe takes as long.  Before, one CTA took one tile
// with P in shared memory and O folded into registers for every block.  B x T x heads x size, causal: 16 x 1024 x 12 x 64 230 ->
// 73 us (351 TFLOP/s), 2 x 4096 x 32/8 x 128 2060 -> 246 us (1115), 64 x 128 x 16 x 128 100 -> 32 us.  Two threads a row (576
// threads, 96 registers) ran at 107 / 451 us: spills; 168 registers a thread without the hand-over at 82 / 269.
//
// Two tiles of rows in turn, rescaling only when it matters and a share of the exponentials as a polynomial are published ideas: FlashAttention-3
// (Shah et al., 2024) and the descriptions of FlashAttention-4 (2025).  The code and its constants are this file's own.
//
// A mask (bytes, non-zero = attend) is turned into 128 bits a row with coalesced byte loads and ballots, so any stride and alignment
// of its rows will do.  Masked scores become a large finite negative: a row with every key masked attends uniformly
// (keras/src/backend/torch/nn.py:1539).
//
// Every mbarrier wait is bounded (iteration limit + abort flag): on expiry the kernel writes a code to *err, lets its
// outstanding copies land, frees TMEM and returns.
#include "gemm_sm100.cuh"

namespace {
using namespace kbgemm;

struct FlashParams {
  int B, H, Hkv, Tq, Tk;
  float scale_log2;  // softmax scale times log2(e), positive
  int causal;
  float* lse;        // [B, H, Tq] natural-log sum of exponentials of the scaled scores
  int* err;
  const uint8_t* mask;  // null, or element (b, h, q, k) at mask[b * mask_b + h * mask_h + q * mask_q + k]
  long long mask_b, mask_h, mask_q;
  const uint8_t* row_mask;  // with mask: null, or element (b, q) at row_mask[b * row_mask_b + q]; rows at zero see masked keys only
  long long row_mask_b;
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

template <int D, int NT>
struct FlashCfg {
  static constexpr int CH = D / 64;                   // 64-column chunks of the head dimension
  static constexpr int TILE_BYTES = CH * 16384;       // Q, O: [chunk][128 rows][128 B]; K the same; V: [64-key block][chunk][64 keys][128 B]
  static constexpr int RING = NT == 2 ? (D == 128 ? 4 : 8) : (D == 128 ? 2 : 4);  // K0 V0 K1 V1 ...
  static constexpr int SMEM = (NT + RING) * TILE_BYTES + 256;  // dynamic shared memory starts 1024-byte aligned
  static constexpr uint32_t TMEM_COLS = NT == 2 ? 512 : 256;   // S per tile (128 columns; P in its first 64), then O per tile (D)
  // NT = 2 adds a whole warpgroup for the TMA and MMA warps, so that it can hand registers to the softmax warps
  static constexpr int THREADS_ = NT == 2 ? 384 : 192;
};

__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// 2^x of two values on the FMA pipe, for the share of the exponentials that the special-function pipe has no time for.
// x = n + f with n the nearest integer (the sum with 1.5 * 2^23 leaves n in the low bits), 2^f on [-1/2, 1/2] by a polynomial of
// degree 5 with the least maximum relative error (a linear program over 4000 Chebyshev points gives its coefficients, rounded to float32;
// 2.1e-7 in float32, as the hardware's own approximation), n added to the exponent.  x is at
// most RESCALE_LOG2; below -126 the result is held at 2^-126, which is nothing beside a row sum of at least 2^-8.
__device__ __forceinline__ void exp2_poly2(uint64_t x2, float& y0, float& y1) {
  float x0, x1;
  unpack_f32x2(x2, x0, x1);
  const uint64_t x = pack_f32x2(fmaxf(x0, -126.f), fmaxf(x1, -126.f));
  const uint64_t t = add_f32x2(x, pack_f32x2(12582912.f, 12582912.f));  // n in the low bits
  const uint64_t n = add_f32x2(t, pack_f32x2(-12582912.f, -12582912.f));
  const uint64_t f = fma_f32x2(n, pack_f32x2(-1.f, -1.f), x);
  uint64_t y = fma_f32x2(pack_f32x2(0.001327647129073739f, 0.001327647129073739f), f, pack_f32x2(0.009675540961325169f, 0.009675540961325169f));
  y = fma_f32x2(y, f, pack_f32x2(0.05550713092088699f, 0.05550713092088699f));
  y = fma_f32x2(y, f, pack_f32x2(0.24022120237350464f, 0.24022120237350464f));
  y = fma_f32x2(y, f, pack_f32x2(0.6931469440460205f, 0.6931469440460205f));
  y = fma_f32x2(y, f, pack_f32x2(1.0000001192092896f, 1.0000001192092896f));
  float t0, t1;
  unpack_f32x2(t, t0, t1);
  unpack_f32x2(y, y0, y1);
  y0 = __uint_as_float(__float_as_uint(y0) + (__float_as_uint(t0) << 23));
  y1 = __uint_as_float(__float_as_uint(y1) + (__float_as_uint(t1) << 23));
}
constexpr int POLY_EVERY = 4;           // one pair of exponentials in four

constexpr float MASKED = -1e30f;        // of a score, before scaling: finite, so that a row of nothing else is uniform
constexpr float RESCALE_LOG2 = 8.f;

template <int D, int NT, bool MASK>
__global__ void __launch_bounds__(FlashCfg<D, NT>::THREADS_, NT == 2 ? 1 : 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                 const __grid_constant__ CUtensorMap map_o, const FlashParams p) {
  using C = FlashCfg<D, NT>;
  constexpr int TILE = C::TILE_BYTES, RING = C::RING;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  if (base & 1023u) {  // the 128-byte swizzle needs 1024-byte aligned tiles; without static shared memory the window starts aligned
    if (threadIdx.x == 0 && p.err) atomicExch(p.err, 30);
    return;
  }
  const uint32_t sQ = base, sKV = sQ + NT * TILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + (NT + RING) * TILE);
  const uint32_t bar_base = sKV + RING * TILE;
  const uint32_t q_bar = bar_base;
  auto kv_full = [&](int s) { return bar_base + 8u * (1 + s); };
  auto kv_empty = [&](int s) { return bar_base + 8u * (1 + RING + s); };
  auto s_full = [&](int i) { return bar_base + 8u * (1 + 2 * RING + i); };
  auto p_ready = [&](int n) { return bar_base + 8u * (1 + 2 * RING + NT + n); };  // tile i: 2i its first 64 keys, 2i + 1 the rest
  auto o_done = [&](int i) { return bar_base + 8u * (1 + 2 * RING + 3 * NT + i); };
  constexpr int N_BARS = 1 + 2 * RING + 4 * NT;
  static_assert(N_BARS * 8 + 8 <= 256, "barrier area");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + N_BARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the longest rows of a causal mask first: the last wave is then made of short ones
  const int groups = p.H * p.B, n_q = (p.Tq + 128 * NT - 1) / (128 * NT);
  const int q0 = (n_q - 1 - (int)(blockIdx.x / groups)) * 128 * NT;
  const int h = (int)(blockIdx.x % groups) % p.H, b = (int)(blockIdx.x % groups) / p.H;
  const int hkv = h / (p.H / p.Hkv);
  // key blocks of tile i; a tile that starts beyond the last query has none
  const int all_blocks = (p.Tk + 127) / 128;
  auto blocks_of = [&](int i) {
    const int first = q0 + i * 128;
    if (first >= p.Tq) return 0;
    return p.causal ? min(all_blocks, first / 128 + 1) : all_blocks;
  };
  const int n_blocks = max(blocks_of(0), NT == 2 ? blocks_of(1) : 0);

  if (threadIdx.x == 0) {
    mbar_init(q_bar, 1);
    for (int s = 0; s < RING; ++s) {
      mbar_init(kv_full(s), 1);
      mbar_init(kv_empty(s), 1);
    }
    for (int i = 0; i < NT; ++i) {
      mbar_init(s_full(i), 1);
      mbar_init(p_ready(2 * i), 4);
      mbar_init(p_ready(2 * i + 1), 4);
      mbar_init(o_done(i), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4 * NT + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(C::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  auto tmem_S = [&](int i) { return tmem_base + (uint32_t)(i * 128); };
  auto tmem_O = [&](int i) { return tmem_base + (uint32_t)(NT * 128 + i * D); };

  // NT = 2: 384 threads x 168 registers at launch = 256 x 224 + 128 x 56
  if (warp < 4 * NT) {
    if constexpr (NT == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // ------------------------------------------------------------------ softmax and output, one thread per query row
    const int i = warp >> 2, q = warp & 3;
    const int row = q * 32 + lane, first = q0 + i * 128, qi = first + row;
    const int nb = blocks_of(i);
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const uint32_t tS = tmem_base + (uint32_t)(i * 128) + lane_base, tO = tmem_base + (uint32_t)(NT * 128 + i * D) + lane_base;
    float m = -INFINITY;  // maximum that P is relative to, scaled to log2
    uint64_t l2[2] = {0, 0};
    bool ok = true;
    for (int j = 0; j < nb; ++j) {
      const int k0 = j * 128;
      uint32_t keep[4];
      if constexpr (MASK) {  // this row's 128 bits, while the score product runs
        const uint8_t* mb = p.mask + (long long)b * p.mask_b + (long long)h * p.mask_h;
        if (p.mask_q == 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int k = k0 + c * 32 + lane;
            keep[c] = __ballot_sync(0xffffffffu, k < p.Tk && mb[k] != 0);
          }
        } else {
#pragma unroll 1
          for (int r0 = 0; r0 < 32; r0 += 8) {
            uint8_t v[8][4];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int qr = min(first + q * 32 + r0 + r, p.Tq - 1);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const int k = k0 + c * 32 + lane;
                v[r][c] = k < p.Tk ? mb[(long long)qr * p.mask_q + k] : 0;
              }
            }
#pragma unroll
            for (int r = 0; r < 8; ++r)
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint32_t bits = __ballot_sync(0xffffffffu, v[r][c] != 0);
                if (lane == r0 + r) keep[c] = bits;
              }
          }
        }
        if (p.row_mask != nullptr && p.row_mask[(long long)b * p.row_mask_b + min(qi, p.Tq - 1)] == 0) keep[0] = keep[1] = keep[2] = keep[3] = 0;
      }
      ok = mbar_wait(s_full(i), j & 1, abort_flag);
      if (!ok) break;
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t r[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + (uint32_t)(c * 32), r + c * 32);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if constexpr (MASK) {
#pragma unroll
        for (int e = 0; e < 128; ++e)
          if (!(keep[e >> 5] >> (e & 31) & 1u)) r[e] = __float_as_uint(MASKED);
      }
      if (k0 + 127 >= p.Tk || (p.causal && k0 + 127 > first)) {
        const int last = p.causal ? min(p.Tk - 1, qi) - k0 : p.Tk - 1 - k0;  // last key of this block that the row may see
#pragma unroll
        for (int e = 0; e < 128; ++e)
          if (e > last) r[e] = __float_as_uint(-INFINITY);
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < 128; e += 8)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx[c] = max_nan(mx[c], max_nan(__uint_as_float(r[e + c]), __uint_as_float(r[e + 4 + c])));
      const float m_new = max_nan(m, max_nan(max_nan(mx[0], mx[1]), max_nan(mx[2], mx[3])) * p.scale_log2);
      l2[0] = add_f32x2(l2[0], pack_f32x2(m_new - m_new, 0.f));  // a NaN or infinite score makes the row NaN, whichever way its exponential goes
      const bool grow = m_new > m + RESCALE_LOG2;  // the first block included: m is -inf
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = grow ? exp2f(m - m_new) : 1.f;
        if (grow) m = m_new;
        const uint64_t a2 = pack_f32x2(alpha, alpha);
        l2[0] = fma_f32x2(l2[0], a2, 0);
        l2[1] = fma_f32x2(l2[1], a2, 0);
        if (j > 0) {  // S(j) is full, so P V of the block before has been added
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tmem_ld16(tO + (uint32_t)(c * 16), o);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st16(tO + (uint32_t)(c * 16), o);
          }
        }
      }
      // So far only masked keys: each counts alike.  The difference of two roundings of so large a product would not be zero, so
      // such rows scale their scores to nothing instead (-inf, a key that is not there, stays what it is).
      const bool blank = MASK && m < 0.5f * MASKED * p.scale_log2;
      const float scale = blank ? 1e-37f : p.scale_log2, m_use = blank ? 0.f : m;
      const uint64_t scale2 = pack_f32x2(scale, scale), minus2 = pack_f32x2(-m_use, -m_use);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float x0, x1;
          const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(r[c * 32 + 2 * e]), __uint_as_float(r[c * 32 + 2 * e + 1])), scale2, minus2);
          if (e % POLY_EVERY == POLY_EVERY - 1) {
            exp2_poly2(x2, x0, x1);
          } else {
            unpack_f32x2(x2, x0, x1);
            x0 = exp2f(x0);
            x1 = exp2f(x1);
          }
          l2[e & 1] = add_f32x2(l2[e & 1], pack_f32x2(x0, x1));
          const __nv_bfloat162 pr = __floats2bfloat162_rn(x0, x1);
          w[e] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        tmem_st16(tS + (uint32_t)(c * 16), w);
        if (c & 1) {  // 64 keys are there: P V may start on them
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(p_ready(2 * i + (c >> 1)));
        }
      }
    }
    if (ok && nb > 0) {
      ok = mbar_wait(o_done(i), 0, abort_flag);
      __syncwarp();
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float la, lb, lc, ld;
        unpack_f32x2(l2[0], la, lb);
        unpack_f32x2(l2[1], lc, ld);
        const float l = (la + lb) + (lc + ld);
        const float inv_l = l == 0.f ? 0.f : 1.f / l;
        // every product of this tile has completed: its Q is free, O is staged there
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + (uint32_t)(c * 32), o);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const uint32_t chunk = sQ + (uint32_t)(i * TILE + (c >> 1) * 16384) + (uint32_t)row * 128u;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(o[u * 8 + e]) * inv_l;
            const bf16x8 pk = pack8(v);
            const uint4 w = *reinterpret_cast<const uint4*>(&pk);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(chunk + (((uint32_t)((c & 1) * 4 + u) ^ (uint32_t)(row & 7)) << 4)), "r"(w.x),
                         "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && first + q * 32 < p.Tq) {
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tma_store_4d(&map_o, sQ + (uint32_t)(i * TILE + c * 16384) + (uint32_t)(q * 32) * 128u, c * 64, first + q * 32, h, b);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the writes land before the grid ends
        }
        if (qi < p.Tq && p.lse != nullptr)
          p.lse[((long long)b * p.H + h) * p.Tq + qi] = (l != 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    }
    if (!ok) {
      if (lane == 0 && p.err) atomicExch(p.err, 33);
      *abort_flag = 1;
    }
  } else {
    if constexpr (NT == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 4 * NT) {
      // ------------------------------------------------------------------ TMA producer
      if (elect_one()) {
        mbar_expect_tx(q_bar, NT * TILE);
#pragma unroll
        for (int i = 0; i < NT; ++i)  // rows beyond the last query arrive as zeros
#pragma unroll
          for (int c = 0; c < C::CH; ++c) tma_load_4d(sQ + i * TILE + c * 16384, &map_q, q_bar, c * 64, q0 + i * 128, h, b);
        bool ok = true;
        int issued = 0;
        for (int n = 0; n < 2 * n_blocks; ++n) {
          const int s = n % RING, k0 = (n >> 1) * 128;
          ok = mbar_wait(kv_empty(s), ((n / RING) & 1) ^ 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(kv_full(s), TILE);
          const uint32_t dst = sKV + s * TILE;
          if ((n & 1) == 0) {
#pragma unroll
            for (int c = 0; c < C::CH; ++c) tma_load_4d(dst + c * 16384, &map_k, kv_full(s), c * 64, k0, hkv, b);
          } else {
#pragma unroll
            for (int kb = 0; kb < 2; ++kb)
#pragma unroll
              for (int c = 0; c < C::CH; ++c) tma_load_4d(dst + (kb * C::CH + c) * 8192, &map_v, kv_full(s), c * 64, k0 + kb * 64, hkv, b);
          }
          issued = n + 1;
        }
        if (!ok) {
          if (p.err) atomicExch(p.err, 31);
          *abort_flag = 1;
          for (uint32_t spin = 0; spin < (1u << 16); ++spin)
            if (mbar_try_wait(q_bar, 0)) break;
          for (int n = max(0, issued - RING); n < issued; ++n)
            for (uint32_t spin = 0; spin < (1u << 16); ++spin)
              if (mbar_try_wait(kv_full(n % RING), (n / RING) & 1)) break;
        }
      }
    } else if (warp == 4 * NT + 1) {
      // ------------------------------------------------------------------ MMA issuer
      if (elect_one()) {
        const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        auto scores = [&](int i, int s) {
#pragma unroll
          for (int c = 0; c < C::CH; ++c) {
            const uint64_t adesc = make_smem_desc(sQ + i * TILE + c * 16384, false), bdesc = make_smem_desc(sKV + s * TILE + c * 16384, false);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16(tmem_S(i), adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc_s, (c > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(s_full(i));
        };
        auto values = [&](int i, int s, int kb, bool first) {
          const uint64_t bdesc = make_smem_desc(sKV + s * TILE + kb * C::CH * 8192, true);
#pragma unroll
          for (int k = 0; k < 4; ++k)  // 16 keys: 8 columns of packed pairs
            umma_bf16_ts(tmem_O(i), tmem_S(i) + (uint32_t)(kb * 32 + k * 8), bdesc + (uint64_t)((2048u >> 4) * k), idesc_o, (!first || kb > 0 || k > 0) ? 1u : 0u);
        };
        int nb[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) nb[i] = blocks_of(i);
        bool ok = mbar_wait(q_bar, 0, abort_flag) && mbar_wait(kv_full(0), 0, abort_flag);
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int i = 0; i < NT; ++i)
            if (nb[i] > 0) scores(i, 0);
          umma_commit(kv_empty(0));
        }
        for (int j = 0; j < n_blocks && ok; ++j) {
          const int nv = 2 * j + 1, nk = 2 * j + 2;  // ring positions of V(j) and K(j + 1)
          ok = mbar_wait(kv_full(nv % RING), (nv / RING) & 1, abort_flag);
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            if (!ok || j >= nb[i]) continue;
#pragma unroll
            for (int kb = 0; kb < 2; ++kb) {
              if (ok) ok = mbar_wait(p_ready(2 * i + kb), j & 1, abort_flag);  // that half of P(j) is in TMEM, S(j) has been read, O rescaled
              if (!ok) continue;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              values(i, nv % RING, kb, j == 0);
            }
            if (!ok) continue;
            if (j + 1 < nb[i]) {
              ok = mbar_wait(kv_full(nk % RING), (nk / RING) & 1, abort_flag);
              if (!ok) continue;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              scores(i, nk % RING);
            } else {
              umma_commit(o_done(i));
            }
          }
          if (!ok) break;
          umma_commit(kv_empty(nv % RING));
          if (j + 1 < n_blocks) umma_commit(kv_empty(nk % RING));
        }
        if (!ok) {
          if (p.err) atomicExch(p.err, 32);
          *abort_flag = 1;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  if (warp == 4 * NT + 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM_COLS) : "memory");
  }
}

template <int D, int NT, bool MASK>
int launch_flash(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& o, const FlashParams& p, cudaStream_t stream) {
  using C = FlashCfg<D, NT>;
  static bool attr[KB_MAX_DEVICES] = {false};
  if (!kb_allow_smem(flash_fwd_kernel<D, NT, MASK>, C::SMEM, attr)) {
    kb200_set_error("flash_attention: shared-memory limit");
    return -3;
  }
  const long long grid = (long long)((p.Tq + 128 * NT - 1) / (128 * NT)) * p.H * p.B;
  flash_fwd_kernel<D, NT, MASK><<<(unsigned)grid, C::THREADS_, C::SMEM, stream>>>(q, k, v, o, p);
  return 0;
}

template <int D>
int launch_flash_any(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const CUtensorMap& o, const FlashParams& p, cudaStream_t stream) {
  if (p.Tq <= 128)  // a single tile of rows: two such CTAs share an SM
    return p.mask ? launch_flash<D, 1, true>(q, k, v, o, p, stream) : launch_flash<D, 1, false>(q, k, v, o, p, stream);
  return p.mask ? launch_flash<D, 2, true>(q, k, v, o, p, stream) : launch_flash<D, 2, false>(q, k, v, o, p, stream);
}

// 4-D bf16 tensor map over [batch, time, heads, head_dim] storage: dims (head_dim, time, heads, batch).
bool make_map_bthd(CUtensorMap* map, const void* ptr, int D, int T, int H, int B, long long stride_t, long long stride_h, long long stride_b, int box_d,
                   int box_t) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)T, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)stride_t * 2, (cuuint64_t)stride_h * 2, (cuuint64_t)stride_b * 2};
  cuuint32_t box[4] = {(cuuint32_t)box_d, (cuuint32_t)box_t, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

// q, o: [B, Tq, H, D]; k, v: [B, Tk, Hkv, D]; bf16, unit stride on D, the other strides (in elements) multiples of 8 and the
// base pointers 16-byte aligned.  D is 64 or 128, H a multiple of Hkv, scale positive.  lse: [B, H, Tq] fp32 (may be null).
// mask: null, or bytes with unit stride over the keys and the given strides over batch, head and query (0 broadcasts).
// row_mask (with mask): null, or bytes [B, Tq]; a row at zero has every key masked.
KB_API int kb200_flash_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Tq, int Tk, int H, int Hkv, int D,
                                     long long q_st, long long q_sh, long long q_sb, long long k_st, long long k_sh, long long k_sb, long long v_st,
                                     long long v_sh, long long v_sb, long long o_st, long long o_sh, long long o_sb, float scale, int causal,
                                     const uint8_t* mask, long long mask_b, long long mask_h, long long mask_q, const uint8_t* row_mask,
                                     long long row_mask_b, int* err, cudaStream_t stream) {
  if (B <= 0 || Tq <= 0 || Tk <= 0 || H <= 0) return 0;
  if ((D != 64 && D != 128) || Hkv <= 0 || H % Hkv) {
    kb200_set_error("flash_attention_fwd: head_dim must be 64 or 128 and the query heads a multiple of the key/value heads");
    return -2;
  }
  if (!(scale > 0.f) || (long long)((Tq + 127) / 128) * H * B > 0x7fffffffll) {
    kb200_set_error("flash_attention_fwd: the scale must be positive and the grid within range");
    return -2;
  }
  if (mask != nullptr && causal) {
    kb200_set_error("flash_attention_fwd: a mask includes the causal one");
    return -2;
  }
  const long long strides[12] = {q_st, q_sh, q_sb, k_st, k_sh, k_sb, v_st, v_sh, v_sb, o_st, o_sh, o_sb};
  for (int i = 0; i < 12; ++i)
    if (strides[i] % 8) {
      kb200_set_error("flash_attention_fwd: strides must be multiples of 8 elements");
      return -2;
    }
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o) & 15) != 0) {
    kb200_set_error("flash_attention_fwd: base pointers must be 16-byte aligned");
    return -2;
  }
  CUtensorMap map_q, map_k, map_v, map_o;
  bool ok = make_map_bthd(&map_q, q, D, Tq, H, B, q_st, q_sh, q_sb, 64, 128) && make_map_bthd(&map_k, k, D, Tk, Hkv, B, k_st, k_sh, k_sb, 64, 128) &&
            make_map_bthd(&map_v, v, D, Tk, Hkv, B, v_st, v_sh, v_sb, 64, 64) && make_map_bthd(&map_o, o, D, Tq, H, B, o_st, o_sh, o_sb, 64, 32);
  if (!ok) {
    kb200_set_error("flash_attention_fwd: cuTensorMapEncodeTiled failed");
    return -3;
  }
  FlashParams p{B, H, Hkv, Tq, Tk, scale * 1.4426950408889634f, causal, lse, err, mask, mask_b, mask_h, mask_q,
                mask != nullptr ? row_mask : nullptr, row_mask_b};
  const int rc = D == 64 ? launch_flash_any<64>(map_q, map_k, map_v, map_o, p, stream) : launch_flash_any<128>(map_q, map_k, map_v, map_o, p, stream);
  if (rc != 0) return rc;
  KB_CHECK_LAUNCH("flash_attention_fwd");
  return 0;
}
