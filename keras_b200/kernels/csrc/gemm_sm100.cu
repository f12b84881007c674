// bf16 GEMM on 5th-generation tensor cores (tcgen05), Blackwell sm_100a.
//
//   C[M,N] = act(A x B + bias)        fp32 accumulation in tensor memory (TMEM)
//
// Operands are fed by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a 3-stage shared-memory
// ring; one elected thread issues tcgen05.mma (128x128x16 per instruction, cta_group::1) with the
// accumulator in TMEM; four epilogue warps read the accumulator back with tcgen05.ld and apply
// bias / activation / output cast on the way to global memory.  Both operands may be K-major or
// MN-major (set in the UMMA instruction and shared-memory descriptors), which covers the forward
// (X·W), input-gradient (dY·Wᵀ) and weight-gradient (Xᵀ·dY) products of a dense layer without any
// transposed copy.  Two CTAs fit per SM (96 KB of operand stages, 128 TMEM columns each) so one
// CTA's epilogue overlaps the other's main loop.
//
// Replaces torch.matmul / cuBLASLt + separate bias and activation kernels
// (keras/src/backend/torch/numpy.py:101-160, keras/src/layers/core/dense.py:238-244).
//
// Every wait on an mbarrier is bounded: on expiry the kernel records a code in `*err`, drains its
// outstanding copies (also bounded), releases TMEM and returns.
#include "gemm_sm100.cuh"

namespace {
using namespace kbgemm;

// STAGES: three leave room for two CTAs an SM, which hide each other's latency; a grid of at most one CTA an SM has no second one and
// takes six, or its loop waits for L2 (600 ns a 64-element K block with three: [2664, 512, 2048] 12.1 -> 10.7 us).
template <int STAGES>
__global__ void __launch_bounds__(THREADS, STAGES == 3 ? 2 : 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ GroupMaps maps, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment is required by the 128-byte swizzle atoms
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base_ptr + STAGES * STAGE_BYTES);
  const uint32_t bar_base = base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  const uint32_t tmem_full_bar = bar_base + 8u * (2 * STAGES);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = p.groups > 1 && !p.sum_k ? p.tile_end[p.groups - 1] : (p.N + BN - 1) / BN;
  const int m0 = (blockIdx.x / n_tiles) * BM;
  int first_tile;
  const int tile_group = group_of_tile(p, blockIdx.x % n_tiles, first_tile);
  const int n0 = ((int)(blockIdx.x % n_tiles) - first_tile) * BN;
  const int k_blocks = p.sum_k ? p.kb_end[p.groups - 1] : (p.K + BK - 1) / BK;
  auto load_block = [&](int kb) {
    int first_kb;
    const int g = tile_group + group_of_block(p, kb, first_kb);
    const CUtensorMap &map_a = maps.a[p.sum_k ? g : 0], &map_b = maps.b[g];
    const int s = kb % STAGES, k0 = (kb - first_kb) * BK;
    const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_TILE_BYTES;
    mbar_expect_tx(full_bar(s), STAGE_BYTES);
    if (p.a_mn_major) {
      tma_load_2d(sa, &map_a, full_bar(s), m0, k0);
      tma_load_2d(sa + 8192, &map_a, full_bar(s), m0 + 64, k0);
    } else {
      tma_load_2d(sa, &map_a, full_bar(s), k0, m0);
    }
    if (p.b_mn_major) {
      tma_load_2d(sb, &map_b, full_bar(s), n0, k0);
      tma_load_2d(sb + 8192, &map_b, full_bar(s), n0 + 64, k0);
    } else {
      tma_load_2d(sb, &map_b, full_bar(s), k0, n0);
    }
  };
  const int first_blocks = min(STAGES, k_blocks);  // loaded ahead of the barrier below, while TMEM is being allocated

  if (threadIdx.x == 0) {
    prefetch_map(&maps.a[0]);
    prefetch_map(&maps.b[0]);
    prefetch_map(&maps.c[0]);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tmem_full_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int kb = 0; kb < first_blocks; ++kb) load_block(kb);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int issued = first_blocks;
      bool ok = true;
      for (int kb = first_blocks; kb < k_blocks && ok; ++kb) {
        ok = mbar_wait(empty_bar(kb % STAGES), ((kb / STAGES) & 1) ^ 1, abort_flag);
        if (!ok) break;
        load_block(kb);
        issued = kb + 1;
      }
      if (!ok) {
        if (p.err) atomicExch(p.err, 1);
        *abort_flag = 1;
        // drain: give copies already issued a bounded time to land before the CTA exits
        const int first = issued > STAGES ? issued - STAGES : 0;
        for (int kb = first; kb < issued; ++kb) {
          const int s = kb % STAGES;
          for (uint32_t it = 0; it < (1u << 16); ++it)
            if (mbar_try_wait(full_bar(s), (kb / STAGES) & 1)) break;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint32_t a_step = p.a_mn_major ? (2048u >> 4) : (32u >> 4);
      const uint32_t b_step = p.b_mn_major ? (2048u >> 4) : (32u >> 4);
      bool ok = true;
      for (int kb = 0; kb < k_blocks; ++kb) {
        const int s = kb % STAGES;
        ok = mbar_wait(full_bar(s), (kb / STAGES) & 1, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_TILE_BYTES;
        const uint64_t adesc = make_smem_desc(sa, p.a_mn_major), bdesc = make_smem_desc(sb, p.b_mn_major);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          umma_bf16(tmem_base, adesc + (uint64_t)(a_step * k), bdesc + (uint64_t)(b_step * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(s));  // frees the stage when these MMAs have read it
      }
      if (ok) {
        umma_commit(tmem_full_bar);
      } else {
        if (p.err) atomicExch(p.err, 2);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const bool ok = mbar_wait(tmem_full_bar, 0, abort_flag);
    if (!ok) {
      if (lane == 0 && p.err) atomicExch(p.err, 3);
      *abort_flag = 1;
    } else {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int q = warp & 3;  // TMEM lane quarter this warp may access
      // every MMA of this CTA's only tile has completed, so the operand ring is free: stage 0 holds the staging buffers
      uint32_t stores = 0;
      store_rows_group(tmem_base + ((uint32_t)(q * 32) << 16), BN, n0, m0 + q * 32, base + (uint32_t)(warp - 2) * 8192u, stores, maps, tile_group, p, lane, 0);
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // staging read out; the writes land before the grid ends
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}


// ---------------------------------------------------------------------------------------------
// Persistent variant for large problems: 128x256 output tiles, four 48 KB operand stages, the whole
// tensor memory (512 columns) split into two 256-column accumulators so that the epilogue of tile i
// overlaps the main loop of tile i+1.  One CTA per SM; tiles are handed out round-robin in an order
__global__ void __launch_bounds__(THREADS, 1)
gemm_bf16_tcgen05_persistent(const __grid_constant__ GroupMaps maps, const GemmParams p) {
  constexpr int BM = v2::BM, BN = v2::BN, BK = v2::BK, STAGES = v2::STAGES, STAGE_BYTES = v2::STAGE_BYTES, A_BYTES = v2::A_BYTES;
  constexpr uint32_t TMEM_COLS = v2::TMEM_COLS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  // after the operand ring: 4 epilogue warps x 2 staging buffers of 4 KB (32 rows x 128 B, swizzled), then the barriers
  const uint32_t stage_out = base + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base_ptr + STAGES * STAGE_BYTES + v2::OUT_BYTES);
  const uint32_t bar_base = stage_out + v2::OUT_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto acc_full_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto acc_empty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 5);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (p.M + BM - 1) / BM, n_tiles = p.groups > 1 && !p.sum_k ? p.tile_end[p.groups - 1] : (p.N + BN - 1) / BN;
  const int split = p.split_k > 1 ? p.split_k : 1;
  const int total_tiles = m_tiles * n_tiles * split;  // work units: (output tile, K slice)
  const int bk = (p.fp8 || p.int8) ? 2 * BK : BK;  // elements per 128-byte K block
  const int k_blocks_all = p.sum_k ? p.kb_end[p.groups - 1] : (p.K + bk - 1) / bk;
  const int kb_per = split > 1 ? p.kb_per_split : k_blocks_all;

  if (threadIdx.x == 0) {
    prefetch_map(&maps.a[0]);
    prefetch_map(&maps.b[0]);
    prefetch_map(&maps.c[0]);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full_bar(a), 1);
      mbar_init(acc_empty_bar(a), 4);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      uint32_t issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        int m0, n0, first_tile, first_kb;
        tile_coords(t / split, m_tiles, n_tiles, m0, n0);
        const int tile_group = group_of_tile(p, n0 / BN, first_tile);
        n0 -= first_tile * BN;
        const int kb0 = (t % split) * kb_per, kb1 = min(kb0 + kb_per, k_blocks_all);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
          mbar_expect_tx(full_bar(s), STAGE_BYTES);
          const int g = tile_group + group_of_block(p, kb, first_kb);
          const CUtensorMap &map_a = maps.a[p.sum_k ? g : 0], &map_b = maps.b[g];
          const int k0 = (kb - first_kb) * bk;
          if (p.a_mn_major) {
            tma_load_2d(sa, &map_a, full_bar(s), m0, k0);
            tma_load_2d(sa + 8192, &map_a, full_bar(s), m0 + 64, k0);
          } else {
            tma_load_2d(sa, &map_a, full_bar(s), k0, m0);
          }
          if (p.b_mn_major) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, &map_b, full_bar(s), n0 + j * 64, k0);
          } else {
            tma_load_2d(sb, &map_b, full_bar(s), k0, n0);
          }
          issued = it + 1;
        }
      }
      if (!ok) {
        if (p.err) atomicExch(p.err, 11);
        *abort_flag = 1;
        const uint32_t first = issued > STAGES ? issued - STAGES : 0;
        for (uint32_t i = first; i < issued; ++i) {
          for (uint32_t spin = 0; spin < (1u << 16); ++spin)
            if (mbar_try_wait(full_bar(i % STAGES), (i / STAGES) & 1)) break;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      // instruction descriptor: fp32 accumulate; operand formats bf16 (kind::f16: 1) or e4m3 / e5m2 (kind::f8f6f4: 0 / 1)
      const uint32_t a_fmt = p.fp8 ? (uint32_t)((p.fp8 - 1) & 1) : 1u, b_fmt = p.fp8 ? (uint32_t)(((p.fp8 - 1) >> 1) & 1) : 1u;
      // kind::i8: accumulator format 2 (s32), operand format 1 (signed 8-bit)
      const uint32_t idesc = p.int8 ? ((2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24))
                                    : ((1u << 4) | (a_fmt << 7) | (b_fmt << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                                       ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24));
      const uint32_t a_step = p.a_mn_major ? (2048u >> 4) : (32u >> 4);
      const uint32_t b_step = p.b_mn_major ? (2048u >> 4) : (32u >> 4);
      uint32_t it = 0, local = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
        const uint32_t acc = local & 1;
        ok = mbar_wait(acc_empty_bar(acc), ((local >> 1) & 1) ^ 1, abort_flag);  // epilogue has drained this accumulator
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + acc * (uint32_t)BN;
        const int kb0 = (t % split) * kb_per, kb1 = min(kb0 + kb_per, k_blocks_all);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(full_bar(s), (it / STAGES) & 1, abort_flag);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
          const uint64_t adesc = make_smem_desc(sa, p.a_mn_major), bdesc = make_smem_desc(sb, p.b_mn_major);
          if (p.int8) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_i8(tmem_d, adesc + (uint64_t)(a_step * k), bdesc + (uint64_t)(b_step * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          } else if (p.fp8) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)  // 32 one-byte elements per instruction: the same 32-byte descriptor step
              umma_f8(tmem_d, adesc + (uint64_t)(a_step * k), bdesc + (uint64_t)(b_step * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          } else {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16(tmem_d, adesc + (uint64_t)(a_step * k), bdesc + (uint64_t)(b_step * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          }
          umma_commit(empty_bar(s));
        }
        if (ok) umma_commit(acc_full_bar(acc));
      }
      if (!ok) {
        if (p.err) atomicExch(p.err, 12);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;
    const uint32_t my_stage = stage_out + (uint32_t)(warp - 2) * 8192u;
    uint32_t local = 0, stores = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
      int m0, n0, first_tile;
      tile_coords(t / split, m_tiles, n_tiles, m0, n0);
      const int tile_group = group_of_tile(p, n0 / BN, first_tile);
      n0 -= first_tile * BN;
      const uint32_t acc = local & 1;
      ok = mbar_wait(acc_full_bar(acc), (local >> 1) & 1, abort_flag);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_row = tmem_base + acc * (uint32_t)BN + ((uint32_t)(q * 32) << 16);
      store_rows_group(tmem_row, BN, n0, m0 + q * 32, my_stage, stores, maps, tile_group, p, lane, t % split);
      // this warp has finished reading the accumulator: hand it back to the MMA issuer
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty_bar(acc));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // staging read out; the writes land before the grid ends
    if (!ok) {
      if (lane == 0 && p.err) atomicExch(p.err, 13);
      *abort_flag = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(v2::TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// CTA-pair variant (cta_group::2): two CTAs of a cluster compute one 256 x 256 tile.  Each holds its own 128 rows of A, half of
// the B tile and the accumulator of its 128 rows; the even CTA issues the MMAs for both.
//
// What bounds the one-CTA kernel is operand traffic: a 128 x 256 tile moves 48 KB from L2 into shared memory for every 512
// tensor-pipe cycles (96 B/clk/SM), more than L2 delivers.  A pair shares B, so the same tile costs 32 KB a CTA (64 B/clk/SM),
// and the smaller stages leave room for eight epilogue warps.
namespace v3 {
constexpr int BM = 128, BN = 256, BK = 64, STAGES = 5;  // BM: rows of one CTA; BN: columns of the pair
constexpr int EPI_WARPS = 8, PAIR_THREADS = 64 + 32 * EPI_WARPS;
constexpr int A_BYTES = BM * BK * 2;
constexpr int OUT_BYTES = EPI_WARPS * 2 * 4096;
constexpr int STAGE_BYTES = A_BYTES + (BN / 2) * BK * 2;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + OUT_BYTES + 1024 + 256;
constexpr uint32_t TMEM_COLS = 2 * BN;  // two accumulators: the epilogue of a tile overlaps the main loop of the next
constexpr int GROUP_M = 8;  // row tiles of 256 side by side: 74 pairs then work on a square patch of the output (4 and 16 measure the same or up to 8 % slower)
}  // namespace v3

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `bar` may be the peer's barrier (a shared::cluster address); the data always lands in this CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs once the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 1023u) == 1023u && *abort_flag) return false;
  }
  return false;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(v3::PAIR_THREADS, 1)
gemm_bf16_tcgen05_pair(const __grid_constant__ GroupMaps maps, const GemmParams p) {
  constexpr int BM = v3::BM, BN = v3::BN, BK = v3::BK, STAGES = v3::STAGES, A_BYTES = v3::A_BYTES, STAGE_BYTES = v3::STAGE_BYTES;
  constexpr uint32_t TMEM_COLS = v3::TMEM_COLS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t stage_out = base + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base_ptr + STAGES * STAGE_BYTES + v3::OUT_BYTES);
  const uint32_t bar_base = stage_out + v3::OUT_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };              // even CTA's is used: bytes of both CTAs
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };  // each CTA its own, signalled by the MMA commit
  auto acc_full_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto acc_empty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };  // even CTA's is used
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 5);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int m_tiles = (p.M + 2 * BM - 1) / (2 * BM), n_tiles = p.groups > 1 && !p.sum_k ? p.tile_end[p.groups - 1] : (p.N + BN - 1) / BN;
  const int split = p.split_k > 1 ? p.split_k : 1;
  const int total_tiles = m_tiles * n_tiles * split;
  const int k_blocks_all = p.sum_k ? p.kb_end[p.groups - 1] : (p.K + BK - 1) / BK;
  const int kb_per = split > 1 ? p.kb_per_split : k_blocks_all;
  auto coords = [&](int t, int& m0, int& n0, int& g) {
    const int per_group = v3::GROUP_M * n_tiles;
    const int patch = t / per_group, first_m = patch * v3::GROUP_M;
    const int rows = min(v3::GROUP_M, m_tiles - first_m);
    const int r = t - patch * per_group;
    m0 = (first_m + r % rows) * (2 * BM);
    int first_tile;
    g = group_of_tile(p, r / rows, first_tile);
    n0 = (r / rows - first_tile) * BN;
  };

  if (threadIdx.x == 0) {
    prefetch_map(&maps.a[0]);
    prefetch_map(&maps.b[0]);
    prefetch_map(&maps.c[0]);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full_bar(a), 1);
      mbar_init(acc_empty_bar(a), 2 * v3::EPI_WARPS);  // one arrival per epilogue warp of both CTAs
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  cluster_sync_all();  // the peer signals this CTA's barriers: they must be initialised first
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (each CTA loads its half of the stage)
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += pairs) {
        int m0, n0, tile_group, first_kb;
        coords(t / split, m0, n0, tile_group);
        m0 += rank * BM;
        n0 += rank * (BN / 2);
        const int kb0 = (t % split) * kb_per, kb1 = min(kb0 + kb_per, k_blocks_all);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
          // The even CTA announces the bytes of both halves.  The odd CTA's copies may complete first: the phase cannot end
          // before the announcement, which is its only arrival.
          if (rank == 0) mbar_expect_tx(full_bar(s), 2 * STAGE_BYTES);
          const uint32_t bar = map_to_rank(full_bar(s), 0);
          const int g = tile_group + group_of_block(p, kb, first_kb);
          const CUtensorMap &map_a = maps.a[p.sum_k ? g : 0], &map_b = maps.b[g];
          const int k0 = (kb - first_kb) * BK;
          if (p.a_mn_major) {
            tma_load_2d_pair(sa, &map_a, bar, m0, k0);
            tma_load_2d_pair(sa + 8192, &map_a, bar, m0 + 64, k0);
          } else {
            tma_load_2d_pair(sa, &map_a, bar, k0, m0);
          }
          if (p.b_mn_major) {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(sb + j * 8192, &map_b, bar, n0 + j * 64, k0);
          } else {
            tma_load_2d_pair(sb, &map_b, bar, k0, n0);
          }
        }
      }
      // Every stage this CTA filled has to be released before it may leave: the releases are remote arrivals on its barriers, and
      // they say that its copies have landed.
      const uint32_t first = it > (uint32_t)STAGES ? it - STAGES : 0;
      for (uint32_t i = first; i < it && ok; ++i) ok = mbar_wait(empty_bar(i % STAGES), (i / STAGES) & 1, abort_flag);
      if (!ok) {
        if (p.err) atomicExch(p.err, 21);
        *abort_flag = 1;
        for (int i = 0; i < 1024; ++i) __nanosleep(1000);  // about a millisecond for the copies in flight
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA, for both)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
      const uint32_t a_step = p.a_mn_major ? (2048u >> 4) : (32u >> 4);
      const uint32_t b_step = p.b_mn_major ? (2048u >> 4) : (32u >> 4);
      uint32_t it = 0, local = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += pairs, ++local) {
        const uint32_t acc = local & 1;
        ok = mbar_wait_cluster(acc_empty_bar(acc), ((local >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + acc * (uint32_t)BN;
        const int kb0 = (t % split) * kb_per, kb1 = min(kb0 + kb_per, k_blocks_all);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait_cluster(full_bar(s), (it / STAGES) & 1, abort_flag);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
          const uint64_t adesc = make_smem_desc(sa, p.a_mn_major), bdesc = make_smem_desc(sb, p.b_mn_major);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(tmem_d, adesc + (uint64_t)(a_step * k), bdesc + (uint64_t)(b_step * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit_pair(empty_bar(s));
        }
        if (ok) umma_commit_pair(acc_full_bar(acc));
      }
      if (!ok) {
        if (p.err) atomicExch(p.err, 22);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9): lane quarter and column half
    const int q = warp & 3, half = (warp - 2) >> 2;
    const uint32_t my_stage = stage_out + (uint32_t)(warp - 2) * 8192u;
    uint32_t local = 0, stores = 0;
    bool ok = true;
    for (int t = pair; t < total_tiles && ok; t += pairs, ++local) {
      int m0, n0, tile_group;
      coords(t / split, m0, n0, tile_group);
      const uint32_t acc = local & 1;
      ok = mbar_wait_cluster(acc_full_bar(acc), (local >> 1) & 1, abort_flag);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_row = tmem_base + acc * (uint32_t)BN + (uint32_t)(half * (BN / 2)) + ((uint32_t)(q * 32) << 16);
      store_rows_group(tmem_row, BN / 2, n0 + half * (BN / 2), m0 + rank * BM + q * 32, my_stage, stores, maps, tile_group, p, lane, t % split);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_rank(acc_empty_bar(acc), 0));
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // staging read out; the writes land before the grid ends
    if (!ok) {
      if (lane == 0 && p.err) atomicExch(p.err, 23);
      *abort_flag = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  cluster_sync_all();  // the peer's MMAs read this CTA's shared memory and write its TMEM; its epilogue arrives on these barriers
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}
}  // namespace


// C[M,N] = act(op(A) op(B) + bias).
//   a_mn_major = 0: A stored [M, K] row-major (pitch lda);  1: A stored [K, M] row-major (pitch lda)
//   b_mn_major = 0: B stored [N, K] row-major (pitch ldb);  1: B stored [K, N] row-major (pitch ldb)
// Requirements: bf16 operands, 16-byte aligned base pointers, pitches multiples of 8 elements;
// C bf16 (out_fp32 = 0) or fp32, ldc multiple of 8 (bf16) / 4 (fp32).  `err` is an int in device
// memory that receives a non-zero code if a bounded wait expires (0 otherwise untouched).
//
// split_k > 1 (persistent kernel only): the K range is cut into `split_k` slices that run as separate work units and
// add their fp32 partial tiles into C with TMA reduce stores; C must be fp32 and zero on entry, bias/act must be off.
// split_k < 0: |split_k| slices and the product is ADDED to what C holds (fp32 gradient accumulation in place).
//
// `variant`: 0 picks one (gemm_variant below); 1: one 128x128 tile a CTA; 2: persistent 128x256 tiles; 3: CTA pairs
// with 256x256 tiles.
enum { GV_AUTO = 0, GV_TILE = 1, GV_PERSISTENT = 2, GV_PAIR256 = 3 };

// Which kernel: work units (output tiles x K slices) against the slots that run at once.  A pair's tile is two SMs' worth of the
// one-CTA kernel's, so both take the same number of waves unless M ends in half a pair, and a wave of pairs is the quicker one
// wherever it was measured: [16384, 50264, 768] 1357 -> 1117 us, [16384, 768, 50264] 1467 -> 1104, weight gradient
// [768, 50264, 16384] 1132 -> 904, [8192, 14336, 4096] 698 -> 636, [768, 3072, 16384] in two slices 70 -> 64.  Below nine tenths of
// a wave of pairs the smaller tiles fill the chip better ([512, 2048, 2664] in four slices: 17.5 us against 19.4).
static int gemm_variant(int M, int N, int split_k, int sms) {
  const long long t1 = (long long)((M + 127) / 128) * ((N + 255) / 256) * split_k, t2 = (long long)((M + 255) / 256) * ((N + 255) / 256) * split_k;
  const long long pairs = sms / 2;
  if (M > 128 && N > 128 && t2 * 10 >= pairs * 9 && (t2 + pairs - 1) / pairs <= (t1 + sms - 1) / sms) return GV_PAIR256;
  if (split_k > 1) return GV_PERSISTENT;
  return N > 128 && t1 >= sms / 2 ? GV_PERSISTENT : GV_TILE;
}

// One product of a launch (see GemmParams::groups).
struct GemmOperands {
  const void *a, *b;
  void* c;
  const void* bias;
  int N, K;
  long long lda, ldb, ldc;
};

// slices_apart: C holds the result of each slice, one below the other, `slice_pitch(M)` rows apart; the number of them comes back in *slices.
static long long slice_pitch(int M) { return (M + 31ll) / 32 * 32; }
static int gemm_launch(const GemmOperands* ops, int groups, int sum_k, int M, int a_mn_major, int b_mn_major, int act, int out_fp32, int bias_bf16, int split_k,
                       int variant, int* err, cudaStream_t stream, int* slices_apart = nullptr) {
  const int accumulate = split_k < 0 ? 1 : 0;
  if (split_k < 0) split_k = -split_k;
  long long columns = 0, k_blocks = 0;  // column tiles are counted per product below
  for (int g = 0; g < groups; ++g) {
    const GemmOperands& o = ops[g];
    if ((split_k > 1 || accumulate) && (!out_fp32 || o.bias != nullptr || act != ACT_NONE)) {
      kb200_set_error("gemm_bf16: split-K needs an fp32 output without bias or activation");
      return -4;
    }
    if ((o.lda % 8) || (o.ldb % 8) || (((uintptr_t)o.a | (uintptr_t)o.b) & 15) || (((uintptr_t)o.c) & 15) || (o.ldc % (out_fp32 ? 4 : 8))) {
      kb200_set_error("gemm_bf16: operands must be 16-byte aligned with pitches that are multiples of 8 elements");
      return -2;
    }
    if (groups > 1 && (sum_k ? o.K % BK || o.N != ops[0].N : o.K != ops[0].K)) {
      kb200_set_error("gemm_bf16: products side by side share K, summed ones share N and have K in whole blocks");
      return -2;
    }
    columns += o.N;
    k_blocks += (o.K + BK - 1) / BK;
  }
  if (sum_k || groups == 1) columns = ops[0].N;
  if (!sum_k) k_blocks = (ops[0].K + BK - 1) / BK;
  const int sm_count = kb_sm_count();
  int kb_per_split = 0;
  if (split_k > 1) {
    if (split_k > k_blocks) split_k = (int)k_blocks;
    kb_per_split = (int)((k_blocks + split_k - 1) / split_k);
    split_k = (int)((k_blocks + kb_per_split - 1) / kb_per_split);  // every slice holds at least one K block
  }
  if (split_k < 1) split_k = 1;
  if (variant == GV_AUTO) variant = gemm_variant(M, (int)(columns > 0x7fffffff ? 0x7fffffff : columns), split_k, sm_count);
  if (split_k > 1 && variant == GV_TILE) variant = GV_PERSISTENT;
  const int tile_m = variant == GV_PAIR256 ? 256 : 128, tile_n = variant == GV_TILE ? 128 : 256;
  // rows of B's box: the N range one CTA loads
  const int bn = variant == GV_PERSISTENT ? 256 : 128;
  GroupMaps maps;
  GemmParams p{ops[0].c, bias_bf16 ? nullptr : (const float*)ops[0].bias, M, ops[0].N, ops[0].K, ops[0].ldc, a_mn_major, b_mn_major, act, out_fp32, err, split_k, kb_per_split};
  p.accumulate = accumulate;
  if (slices_apart != nullptr) {
    *slices_apart = split_k;
    p.slice_rows = split_k > 1 ? (int)slice_pitch(M) : 0;
  }
  p.groups = groups;
  p.sum_k = sum_k;
  // with several products this only says which type the biases are
  p.bias16 = bias_bf16 ? (const __nv_bfloat16*)(groups > 1 ? ops[0].a : ops[0].bias) : nullptr;
  int tiles_n = 0, blocks = 0;
  bool ok = true;
  for (int g = 0; g < 3; ++g) {
    if (g >= groups) {
      maps.a[g] = maps.a[0], maps.b[g] = maps.b[0], maps.c[g] = maps.c[0];
      continue;
    }
    const GemmOperands& o = ops[g];
    ok = ok && (a_mn_major ? make_map(&maps.a[g], o.a, M, o.K, o.lda, 64, BK) : make_map(&maps.a[g], o.a, o.K, M, o.lda, BK, BM));
    ok = ok && (b_mn_major ? make_map(&maps.b[g], o.b, o.N, o.K, o.ldb, 64, BK) : make_map(&maps.b[g], o.b, o.K, o.N, o.ldb, BK, bn));
    ok = ok && make_map(&maps.c[g], o.c, o.N, p.slice_rows ? (int)(slice_pitch(M) * split_k) : M, o.ldc, out_fp32 ? 32 : 64, 32, out_fp32 != 0);
    tiles_n += (o.N + tile_n - 1) / tile_n;
    blocks += (o.K + BK - 1) / BK;
    p.tile_end[g] = tiles_n, p.width[g] = o.N, p.kb_end[g] = blocks, p.bias_of[g] = o.bias;
  }
  if (sum_k) tiles_n = p.tile_end[0];
  if (!ok) {
    kb200_set_error("gemm_bf16: cuTensorMapEncodeTiled failed");
    return -3;
  }
  constexpr int LONG = 6;
  constexpr int smem_v1 = SMEM_BYTES, smem_long = SMEM_BYTES + (LONG - STAGES) * STAGE_BYTES;
  static bool attr_long[KB_MAX_DEVICES] = {false};
  static bool attr_v1[KB_MAX_DEVICES] = {false}, attr_v2[KB_MAX_DEVICES] = {false}, attr_v3[KB_MAX_DEVICES] = {false};
  const bool allowed = variant == GV_TILE         ? kb_allow_smem(gemm_bf16_tcgen05_kernel<STAGES>, smem_v1, attr_v1) &&
                                                        kb_allow_smem(gemm_bf16_tcgen05_kernel<LONG>, smem_long, attr_long)
                       : variant == GV_PERSISTENT ? kb_allow_smem(gemm_bf16_tcgen05_persistent, v2::SMEM_BYTES, attr_v2)
                                                  : kb_allow_smem(gemm_bf16_tcgen05_pair, v3::SMEM_BYTES, attr_v3);
  if (!allowed) {
    kb200_set_error("gemm_bf16: cannot raise the shared-memory limit of the kernel on this device");
    return -3;
  }
  const long long units = (long long)((M + tile_m - 1) / tile_m) * tiles_n * split_k;
  if (variant == GV_TILE) {
    if (units <= sm_count)
      gemm_bf16_tcgen05_kernel<LONG><<<(unsigned)units, THREADS, smem_long, stream>>>(maps, p);
    else
      gemm_bf16_tcgen05_kernel<STAGES><<<(unsigned)units, THREADS, smem_v1, stream>>>(maps, p);
  } else if (variant == GV_PERSISTENT) {
    gemm_bf16_tcgen05_persistent<<<(unsigned)(units < sm_count ? units : sm_count), THREADS, v2::SMEM_BYTES, stream>>>(maps, p);
  } else {
    const int pairs = (int)(units < sm_count / 2 ? units : sm_count / 2);
    gemm_bf16_tcgen05_pair<<<(unsigned)(2 * pairs), v3::PAIR_THREADS, v3::SMEM_BYTES, stream>>>(maps, p);
  }
  KB_CHECK_LAUNCH("gemm_bf16");
  return 0;
}

// `bias_bf16`: the bias holds bf16.
KB_API int kb200_gemm_bf16_run(const void* a, const void* b, void* c, const void* bias, int M, int N, int K, long long lda, long long ldb,
                               long long ldc, int a_mn_major, int b_mn_major, int act, int out_fp32, int bias_bf16, int split_k, int variant, int* err,
                               cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const GemmOperands o{a, b, c, bias, N, K, lda, ldb, ldc};
  return gemm_launch(&o, 1, 0, M, a_mn_major, b_mn_major, act, out_fp32, bias_bf16, split_k, variant, err, stream);
}

namespace {
// out [M, N] = the sum of the slices' results, added in their order and rounded once; four columns a thread
__global__ void __launch_bounds__(256) slice_sum_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out, long long quads, long long step, int slices) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= quads) return;
  const float4* s = reinterpret_cast<const float4*>(part) + i;
  float4 v = *s;
#pragma unroll 4
  for (int k = 1; k < slices; ++k) {
    const float4 q = s[k * step];
    v.x += q.x, v.y += q.y, v.z += q.z, v.w += q.w;
  }
  __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
  reinterpret_cast<uint2*>(out)[i] = *reinterpret_cast<const uint2*>(h);
}
}  // namespace

// Floats of the workspace of kb200_gemm_bf16_slices.
KB_API long long kb200_gemm_slices_floats(int M, int N, int slices) { return slice_pitch(M) * slices * N; }

// C [M, N] (bf16, contiguous, N a multiple of 8) = op(A) op(B) with K in `slices` parts that are added in their order, so that the result does not
// depend on timing.  Slices that add their tiles to C as they come do, and need C cleared and rounded: [2664, 512, 8009] 42.0 us cold, here 39.3.
KB_API int kb200_gemm_bf16_slices(const void* a, const void* b, void* c, float* part, int M, int N, int K, long long lda, long long ldb, int a_mn_major, int b_mn_major,
                                  int slices, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (N % 8 || slices < 2 || slice_pitch(M) * slices > 0x7fffffffll || (((uintptr_t)c | (uintptr_t)part) & 15)) {
    kb200_set_error("gemm_bf16_slices: two slices or more, rows in multiples of 8 columns, 16-byte aligned results");
    return -2;
  }
  const GemmOperands o{a, b, part, nullptr, N, K, lda, ldb, N};
  int made = 1;
  const int rc = gemm_launch(&o, 1, 0, M, a_mn_major, b_mn_major, ACT_NONE, 1, 0, slices, 0, err, stream, &made);
  if (rc != 0) return rc;
  const long long quads = (long long)M * N / 4;
  slice_sum_kernel<<<(unsigned)((quads + 255) / 256), 256, 0, stream>>>(part, (__nv_bfloat16*)c, quads, slice_pitch(M) * N / 4, made);
  KB_CHECK_LAUNCH("slice_sum");
  return 0;
}

// Up to three products in one launch, the fields of GemmOperands one product after the other: pointers (a, b, c, bias), sizes (N, K) and
// pitches (lda, ldb, ldc).  sum_k = 0: C_i = A B_i + bias_i, side by side; sum_k = 1: C = the sum of A_i B_i, added in fp32.  The projections
// of an attention layer, their weight gradients, and the gradient of their common input.
KB_API int kb200_gemm_group(const void* const* pointers, const int* sizes, const long long* pitches, int groups, int sum_k, int M, int a_mn_major, int b_mn_major,
                            int out_fp32, int bias_bf16, int split_k, int variant, int* err, cudaStream_t stream) {
  if (M <= 0) return 0;
  GemmOperands o[3];
  if (groups < 1 || groups > 3) {
    kb200_set_error("gemm_group: one to three products");
    return -2;
  }
  for (int g = 0; g < groups; ++g) {
    o[g] = GemmOperands{pointers[4 * g], pointers[4 * g + 1], const_cast<void*>(pointers[4 * g + 2]), pointers[4 * g + 3], sizes[2 * g], sizes[2 * g + 1],
                        pitches[3 * g], pitches[3 * g + 1], pitches[3 * g + 2]};
    if (o[g].N <= 0 || o[g].K <= 0) {
      kb200_set_error("gemm_group: empty product");
      return -2;
    }
  }
  return gemm_launch(o, groups, groups > 1 ? sum_k : 0, M, a_mn_major, b_mn_major, ACT_NONE, out_fp32, bias_bf16, split_k, variant, err, stream);
}

// C[M,N] = act(alpha * (A x B^T) + bias) with one-byte floating-point operands on kind::f8f6f4 tensor-core instructions.
//   A: [M, K] bytes, row pitch lda bytes;  B: [N, K] bytes, row pitch ldb bytes (both K-major)
//   a_format / b_format: 0 = e4m3, 1 = e5m2;  alpha: device scalar (product of the operands' scales) or null
// Pitches must be multiples of 16 bytes and base pointers 16-byte aligned.  Always runs the persistent kernel.
KB_API int kb200_gemm_fp8(const void* a, const void* b, void* c, const float* bias, const float* alpha, int M, int N, int K, long long lda,
                          long long ldb, long long ldc, int a_format, int b_format, int act, int out_fp32, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 16) || (ldb % 16) || (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) || (ldc % (out_fp32 ? 4 : 8)) || (a_format & ~1) || (b_format & ~1)) {
    kb200_set_error("gemm_fp8: operands must be 16-byte aligned with pitches that are multiples of 16 bytes; formats 0 (e4m3) or 1 (e5m2)");
    return -2;
  }
  GroupMaps maps;
  CUtensorMap &map_a = maps.a[0], &map_b = maps.b[0], &map_c = maps.c[0];
  bool ok = make_map_u8(&map_a, a, K, M, lda, 128, v2::BM) && make_map_u8(&map_b, b, K, N, ldb, 128, v2::BN);
  ok = ok && make_map(&map_c, c, N, M, ldc, out_fp32 ? 32 : 64, 32, out_fp32 != 0);
  if (!ok) {
    kb200_set_error("gemm_fp8: cuTensorMapEncodeTiled failed");
    return -3;
  }
  static bool attr_v2[KB_MAX_DEVICES] = {false};
  if (!kb_allow_smem(gemm_bf16_tcgen05_persistent, v2::SMEM_BYTES, attr_v2)) {
    kb200_set_error("gemm: cannot raise the shared-memory limit of the kernel on this device");
    return -3;
  }
  const int sm_count = kb_sm_count();
  GemmParams p{c, bias, M, N, K, ldc, 0, 0, act, out_fp32, err, 1, 0, 1 + a_format + 2 * b_format, alpha};
  const long long tiles = (long long)((M + v2::BM - 1) / v2::BM) * ((N + v2::BN - 1) / v2::BN);
  gemm_bf16_tcgen05_persistent<<<(unsigned)(tiles < sm_count ? tiles : sm_count), THREADS, v2::SMEM_BYTES, stream>>>(maps, p);
  KB_CHECK_LAUNCH("gemm_fp8");
  return 0;
}

// C[M,N] = act((A x B^T) * row_scale[m] * col_scale[n] + bias) with signed 8-bit operands (kind::i8, int32 accumulation).
//   A: [M, K] int8, row pitch lda bytes;  B: [N, K] int8, row pitch ldb bytes (both K-major)
KB_API int kb200_gemm_i8(const void* a, const void* b, void* c, const float* bias, const float* row_scale, const float* col_scale, int M, int N, int K,
                         long long lda, long long ldb, long long ldc, int act, int out_fp32, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 16) || (ldb % 16) || (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) || (ldc % (out_fp32 ? 4 : 8))) {
    kb200_set_error("gemm_i8: operands must be 16-byte aligned with pitches that are multiples of 16 bytes");
    return -2;
  }
  GroupMaps maps;
  CUtensorMap &map_a = maps.a[0], &map_b = maps.b[0], &map_c = maps.c[0];
  bool ok = make_map_u8(&map_a, a, K, M, lda, 128, v2::BM) && make_map_u8(&map_b, b, K, N, ldb, 128, v2::BN);
  ok = ok && make_map(&map_c, c, N, M, ldc, out_fp32 ? 32 : 64, 32, out_fp32 != 0);
  if (!ok) {
    kb200_set_error("gemm_i8: cuTensorMapEncodeTiled failed");
    return -3;
  }
  static bool attr_v2[KB_MAX_DEVICES] = {false};
  if (!kb_allow_smem(gemm_bf16_tcgen05_persistent, v2::SMEM_BYTES, attr_v2)) {
    kb200_set_error("gemm: cannot raise the shared-memory limit of the kernel on this device");
    return -3;
  }
  const int sm_count = kb_sm_count();
  GemmParams p{c, bias, M, N, K, ldc, 0, 0, act, out_fp32, err, 1, 0, 0, nullptr, 1, row_scale, col_scale};
  const long long tiles = (long long)((M + v2::BM - 1) / v2::BM) * ((N + v2::BN - 1) / v2::BN);
  gemm_bf16_tcgen05_persistent<<<(unsigned)(tiles < sm_count ? tiles : sm_count), THREADS, v2::SMEM_BYTES, stream>>>(maps, p);
  KB_CHECK_LAUNCH("gemm_i8");
  return 0;
}
