// float32 products of few rows on the FMA pipes: C[M, N] = act(op(A) op(B) + bias), or C += op(A) op(B).
//
// The products of a small dense layer have too few output tiles for the chip (16 tiles of 64 x 64 at 128 rows and 512 units), and one CTA a
// tile then walks the whole K range: latency, 7 to 12 us for 0.1 GFLOP.  Here the CTAs of a cluster share K, a tile each, and add their
// partial sums through distributed shared memory in the order of their ranks, so results do not depend on timing.  Bias and rectifier ride
// on the sum, and weight gradients are added where they are kept.  Plain fp32 products and sums throughout.
//
// The step of a classifier of 128 rows, 784 features, 512 units twice and 10 classes: three forward products 12.3 -> 8.5 us each (with their
// rectifiers), two for the inputs' gradients 7.0 -> 5.6, and 58 -> 45 launches in its graph, 167 -> 120 us on the device.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256, MAX_SLICES = 8;
constexpr int AHEAD = 4;         // blocks of K on their way: a slice is some seven blocks long, and each would else cost a latency
constexpr int PITCH = BM + 4;  // floats a row of a tile in shared memory, k-major: rows start on 16 bytes

struct SgemmParams {
  const float* a;
  const float* b;
  float* c;
  const float* bias;
  int M, N, K, slices, k_per;
  long long lda, ldb, ldc;
  int a_vec, b_vec, c_vec;  // rows of the matrix start on 16-byte lines
  int relu, accumulate;
};

// A tile of an operand for one block of K, as a thread holds it between memory and shared memory.
//   ROWS (stored [rows, K]): four consecutive k of one row;  otherwise (stored [K, rows]): four consecutive rows of one k
template <bool ROWS>
struct Fragment {
  float v[4];
  __device__ __forceinline__ void load(const float* p, long long ld, int rows, int K, int r0, int k0, int vec, int tid) {
    const int r = r0 + (ROWS ? tid >> 2 : (tid & 15) * 4), k = k0 + (ROWS ? (tid & 3) * 4 : tid >> 4);
    const float* s = ROWS ? p + (size_t)r * ld + k : p + (size_t)k * ld + r;
    const int left = ROWS ? (r < rows ? K - k : 0) : (k < K ? rows - r : 0);  // values of the four that exist
    if (vec && left >= 4) {
      const float4 q = *reinterpret_cast<const float4*>(s);
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = j < left ? s[j] : 0.f;
    }
  }
  __device__ __forceinline__ void store(float (*t)[PITCH], int tid) const {
    if (ROWS) {
#pragma unroll
      for (int j = 0; j < 4; ++j) t[(tid & 3) * 4 + j][tid >> 2] = v[j];
    } else {
      *reinterpret_cast<float4*>(&t[tid >> 4][(tid & 15) * 4]) = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
};

// A_ROWS: A is stored [M, K] (else [K, M]);  B_ROWS: B is stored [N, K] (else [K, N])
template <bool A_ROWS, bool B_ROWS>
__global__ void __launch_bounds__(THREADS) sgemm_kernel(const SgemmParams p) {
  __shared__ __align__(16) float as[2][BK][PITCH], bs[2][BK][PITCH];
  __shared__ __align__(16) float sums[BM][BN + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int slice = blockIdx.x % p.slices, tile = blockIdx.x / p.slices, n_tiles = (p.N + BN - 1) / BN;
  const int m0 = tile / n_tiles * BM, n0 = tile % n_tiles * BN;
  const int k_begin = slice * p.k_per, k_end = min(p.K, k_begin + p.k_per);
  Fragment<A_ROWS> fa[AHEAD];
  Fragment<B_ROWS> fb[AHEAD];
  float acc[4][4] = {};
#pragma unroll
  for (int d = 0; d < AHEAD; ++d) {
    fa[d].load(p.a, p.lda, p.M, k_end, m0, k_begin + d * BK, p.a_vec, tid);
    fb[d].load(p.b, p.ldb, p.N, k_end, n0, k_begin + d * BK, p.b_vec, tid);
  }
  for (int base = k_begin; base < k_end; base += AHEAD * BK) {
#pragma unroll
    for (int d = 0; d < AHEAD; ++d) {
      const int k0 = base + d * BK;
      if (k0 >= k_end) break;
      const int buf = d & 1;
      fa[d].store(as[buf], tid);
      fb[d].store(bs[buf], tid);
      __syncthreads();  // one a block: the buffer written next was read before the last barrier
      if (k0 + AHEAD * BK < k_end) {
        fa[d].load(p.a, p.lda, p.M, k_end, m0, k0 + AHEAD * BK, p.a_vec, tid);
        fb[d].load(p.b, p.ldb, p.N, k_end, n0, k0 + AHEAD * BK, p.b_vec, tid);
      }
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(&as[buf][k][ty * 4]), y = *reinterpret_cast<const float4*>(&bs[buf][k][tx * 4]);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ys[j], acc[i][j]);
      }
    }
  }
  if (p.slices > 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(&sums[ty * 4 + i][tx * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // this CTA's share of the tile: with one slice each thread's own block, else 64 / slices rows, one row of four columns a thread and turn
  const int share = (BM + p.slices - 1) / p.slices, r_end = min(BM, (slice + 1) * share);
  auto finish = [&](int r, int c, const float* v) {
    const int left = m0 + r < p.M ? p.N - n0 - c : 0;  // columns of the four that exist
    if (left <= 0) return;
    float* out = p.c + (size_t)(m0 + r) * p.ldc + n0 + c;
    float s[4], old[4] = {0.f, 0.f, 0.f, 0.f};
    const bool whole = p.c_vec && left >= 4;
    if (p.accumulate) {
      if (whole) {
        const float4 q = *reinterpret_cast<const float4*>(out);
        old[0] = q.x, old[1] = q.y, old[2] = q.z, old[3] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) old[j] = j < left ? out[j] : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = v[j] + (p.bias != nullptr && j < left ? p.bias[n0 + c + j] : 0.f);
      if (p.relu) s[j] = s[j] <= 0.f ? 0.f : s[j];  // a NaN stays one
      s[j] += old[j];
    }
    if (whole) {
      *reinterpret_cast<float4*>(out) = make_float4(s[0], s[1], s[2], s[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) out[j] = s[j];
    }
  };
  if (p.slices == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) finish(ty * 4 + i, tx * 4, acc[i]);
    return;
  }
  for (int r = slice * share + ty; r < r_end; r += THREADS / 16) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(&sums[r][tx * 4]);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    float4 part[MAX_SLICES];
#pragma unroll
    for (int s = 0; s < MAX_SLICES; ++s) {
      if (s < p.slices) {
        uint32_t peer;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(s));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(part[s].x), "=f"(part[s].y), "=f"(part[s].z), "=f"(part[s].w) : "r"(peer) : "memory");
      }
    }
#pragma unroll
    for (int s = 0; s < MAX_SLICES; ++s)
      if (s < p.slices) v[0] += part[s].x, v[1] += part[s].y, v[2] += part[s].z, v[3] += part[s].w;
    finish(r, tx * 4, v);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // the peers still read these sums
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// dz = dy where the rectified output is positive (0 elsewhere: an infinite gradient at a closed one is zero), or dz = dy without one (then
// not written); db += column sums.  A CTA has 32 columns, its eight warps every eighth row, summed in a fixed order.
__global__ void __launch_bounds__(256) relu_bwd_kernel(const float* __restrict__ dy, const float* __restrict__ out, float* __restrict__ dz, float* __restrict__ db, int M,
                                                       int N, int accumulate) {
  __shared__ float part[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < N) {
#pragma unroll 4
    for (int r = warp; r < M; r += 8) {
      const size_t at = (size_t)r * N + c;
      float g = dy[at];
      if (out != nullptr) {
        g = out[at] > 0.f || out[at] != out[at] ? g : 0.f;
        dz[at] = g;
      }
      s += g;
    }
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < N && db != nullptr) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w][lane];
    db[c] = accumulate ? db[c] + t : t;
  }
}

template <bool A_ROWS, bool B_ROWS>
int launch(const SgemmParams& p, long long tiles, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * p.slices));
  cfg.blockDim = dim3(THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.slices;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, sgemm_kernel<A_ROWS, B_ROWS>, p);
  KB_CHECK_LAUNCH("sgemm");
  return 0;
}

// Weight gradients of layers that see many rows: C[M, N] = A^T B for A [K, M] and B [K, N] of K rows, and B's column sums beside it.
//
// Both operands lie in memory as the FMA loop wants them, k by k, so tiles go to shared memory by asynchronous copies alone and a thread
// forms 8 x 8 sums from four 16-byte reads a k.  K is cut into so many slices that the CTAs fill the chip once; the slices' sums go
// to a workspace (at most 20 MB, mostly met again in L2) and are added in their order by a second launch, which also adds to the gradient
// where it is kept.  Bound by the FMA rate: 256 x 1024 over 6400 rows is 1.68 G products, 46 us at 128 a cycle
// and SM; 77 us with the sums (the library's product 102 and sums 16), 32 x 1024 17 us (51).  The loop runs at 70 % of that rate with 8 x 8
// sums a thread and 16 warps an SM, as it does with 16 x 8 and 8 warps.
constexpr int WN = 128, WK = 16, W_STAGES = 3;
constexpr int w_places(int wm) { return wm == 32 ? 6 : 4; }  // CTAs an SM: shared memory of 31 or 37 KB each, and 128 registers a thread

struct WgradParams {
  const float* a;
  const float* b;
  float* part;  // [slices, M + 1, pitch]: a slice's sums, its column sums in the last row
  int M, N, K, slices, k_per, m_tiles, pitch;
  long long lda, ldb;
  int a_vec, b_vec;  // every row starts on a 16-byte line and holds a multiple of four values
};

__device__ __forceinline__ void copy_async16(uint32_t to, const float* from, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t to, const float* from, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(real ? 4 : 0) : "memory");
}

// WK rows of an operand from row k0, W columns of them from column c0; zeros beyond k_end and beyond its `cols` columns
template <int W, int T>
__device__ __forceinline__ void copy_tile(float* tile, const float* p, long long ld, int cols, int c0, int k0, int k_end, int vec, int tid) {
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(tile);
  if (vec) {
#pragma unroll
    for (int v = tid; v < WK * W / 4; v += T) {
      const int k = v / (W / 4), c = v % (W / 4) * 4;
      const bool real = k0 + k < k_end && c0 + c < cols;
      copy_async16(to + v * 16, real ? p + (size_t)(k0 + k) * ld + c0 + c : p, real);
    }
  } else {
    for (int v = tid; v < WK * W; v += T) {
      const int k = v / W, c = v % W;
      const bool real = k0 + k < k_end && c0 + c < cols;
      copy_async4(to + v * 4, real ? p + (size_t)(k0 + k) * ld + c0 + c : p, real);
    }
  }
}

// A warp has 32 x 64 of a tile, a thread rows {0, 16} + 4 and columns {0, 32} + 4 of it: a warp's reads are 64 and 128 consecutive bytes
template <int WM>
__global__ void __launch_bounds__(WM * 2, w_places(WM)) wgrad_kernel(const WgradParams p) {
  constexpr int T = WM * 2;
  __shared__ __align__(16) float as[W_STAGES][WK][WM], bs[W_STAGES][WK][WN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slice = blockIdx.x % p.slices, tile = blockIdx.x / p.slices;
  const int m0 = tile % p.m_tiles * WM, n0 = tile / p.m_tiles * WN;
  const int k_begin = slice * p.k_per, k_end = min(p.K, k_begin + p.k_per), blocks = (k_end - k_begin + WK - 1) / WK;
  const int rm = (warp >> 1) * 32 + (lane >> 3) * 4, rn = (warp & 1) * 64 + (lane & 7) * 4;
  auto fetch = [&](int i) {
    if (i < blocks) {
      copy_tile<WM, T>(&as[i % W_STAGES][0][0], p.a, p.lda, p.M, m0, k_begin + i * WK, k_end, p.a_vec, tid);
      copy_tile<WN, T>(&bs[i % W_STAGES][0][0], p.b, p.ldb, p.N, n0, k_begin + i * WK, k_end, p.b_vec, tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 acc[8][4] = {};  // pairs of columns: two products an instruction, so that the reads of shared memory find issue slots
  float sums[WN / T] = {};
#pragma unroll
  for (int i = 0; i < W_STAGES - 1; ++i) fetch(i);
  for (int i = 0; i < blocks; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(W_STAGES - 2) : "memory");
    __syncthreads();  // block i is in shared memory, and every thread is done with block i - 1, whose place is filled next
    fetch(i + W_STAGES - 1);
    const float(*x)[WM] = as[i % W_STAGES];
    const float(*y)[WN] = bs[i % W_STAGES];
#pragma unroll
    for (int k = 0; k < WK; ++k) {
      float u[8];
      float2 v[4];
      *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(&x[k][rm]);
      *reinterpret_cast<float4*>(u + 4) = *reinterpret_cast<const float4*>(&x[k][rm + 16]);
      *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(&y[k][rn]);
      *reinterpret_cast<float4*>(v + 2) = *reinterpret_cast<const float4*>(&y[k][rn + 32]);
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = __ffma2_rn(make_float2(u[r], u[r]), v[c], acc[r][c]);
    }
    if (m0 == 0) {
#pragma unroll
      for (int c = 0; c < WN / T; ++c)
#pragma unroll
        for (int k = 0; k < WK; ++k) sums[c] += y[k][c * T + tid];
    }
  }
  float* out = p.part + (size_t)slice * (p.M + 1) * p.pitch;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int m = m0 + rm + (r & 3) + (r >> 2) * 16;
    if (m >= p.M) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (n0 + rn + h * 32 < p.pitch)
        *reinterpret_cast<float4*>(out + (size_t)m * p.pitch + n0 + rn + h * 32) = make_float4(acc[r][h * 2].x, acc[r][h * 2].y, acc[r][h * 2 + 1].x, acc[r][h * 2 + 1].y);
  }
  if (m0 == 0) {
#pragma unroll
    for (int c = 0; c < WN / T; ++c)
      if (n0 + c * T + tid < p.pitch) out[(size_t)p.M * p.pitch + n0 + c * T + tid] = sums[c];
  }
}

// c (+)= the slices' sums, db (+)= those of the last row (db null: left out).  A CTA has 32 quads of columns, its eight warps every eighth
// slice, summed in a fixed order.
__global__ void __launch_bounds__(256) wgrad_sum_kernel(const float* __restrict__ part, float* __restrict__ c, float* __restrict__ db, int M, int N, int pitch, int slices,
                                                        int add, int add_db) {
  __shared__ float4 warps[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quads = pitch / 4, at = blockIdx.x * 32 + lane;
  const bool real = at < (M + (db != nullptr ? 1 : 0)) * quads;
  const float4* s = reinterpret_cast<const float4*>(part) + at;
  const size_t step = (size_t)(M + 1) * quads;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (real) {
#pragma unroll 4
    for (int i = warp; i < slices; i += 8) {
      const float4 q = s[i * step];
      v.x += q.x, v.y += q.y, v.z += q.z, v.w += q.w;
    }
  }
  warps[warp][lane] = v;
  __syncthreads();
  if (warp != 0 || !real) return;
  const int row = at / quads, col = at % quads * 4;
  float* out = row < M ? c + (size_t)row * N + col : db + col;
  const bool more = row < M ? add : add_db;
  float old[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) old[j] = more && col + j < N ? out[j] : 0.f;
#pragma unroll
  for (int w = 1; w < 8; ++w) v.x += warps[w][lane].x, v.y += warps[w][lane].y, v.z += warps[w][lane].z, v.w += warps[w][lane].w;
  const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (col + j < N) out[j] = old[j] + t[j];
}

int wgrad_rows(int M) { return M <= 32 ? 32 : 64; }

// Slices of K, their length a multiple of a block: the cheapest by the CTAs an SM has in turn (33 ns a row of K and full tile; fewer than
// three full CTAs an SM leave the FMA pipes waiting) and by the workspace that is written and read again, among those that run at once.
int wgrad_slices(int M, int N, int K, int* k_per) {
  const int wm = wgrad_rows(M), sms = kb_sm_count(), full = 64 / wm;
  const long long tiles = (long long)((M + wm - 1) / wm) * ((N + WN - 1) / WN);
  int best = 1;
  double least = 1e300;
  for (long long s = 1; s == 1 || (s * tiles <= (long long)sms * w_places(wm) && s <= K / (2 * WK)); ++s) {
    const int rows = (int)(((K + s - 1) / s + WK - 1) / WK * WK);
    if (s > 1 && (long long)rows * (s - 1) >= K) continue;  // no rows for the last
    const long long turn = (s * tiles + sms - 1) / sms;
    const double alone = turn * 1. / full, idle = alone >= 4 ? 1.0 : alone >= 3 ? 1.07 : alone >= 2 ? 1.25 : alone >= 1 ? 2.2 : 2.2 / alone;
    const double ns = turn * (rows + 2. * WK) * 33. / full * idle + s * (M + 1.) * N * 8. / 4000.;
    if (ns < least) least = ns, best = (int)s;
  }
  *k_per = (int)(((K + best - 1) / best + WK - 1) / WK * WK);
  return (K + *k_per - 1) / *k_per;
}
}  // namespace

// C[M, N] = act(op(A) op(B) + bias) in float32.  a_rows: A is [M, K], else [K, M]; b_rows: B is [N, K], else [K, N] (not with A as [K, M]);
// row pitches lda, ldb, ldc.  relu: on the result; accumulate: C += (no bias, no relu).
KB_API int kb200_sgemm(const float* a, const float* b, float* c, const float* bias, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_rows,
                       int b_rows, int relu, int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (!a_rows && b_rows) || (accumulate && (bias != nullptr || relu))) {
    kb200_set_error("sgemm: an empty sum, both operands transposed, or an epilogue on an accumulated result");
    return -2;
  }
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  // K shared by up to eight CTAs while that leaves each two blocks or more and two such CTAs an SM hold all of them
  int slices = 1;
  while (slices < MAX_SLICES && tiles * (slices + 1) <= 2ll * kb_sm_count() && K / (slices + 1) >= 2 * BK) ++slices;
  int k_per = (K + slices - 1) / slices;
  k_per = (k_per + BK - 1) / BK * BK;
  slices = (K + k_per - 1) / k_per;
  if (tiles * slices > 0x7fffffffll) {
    kb200_set_error("sgemm: too many tiles for one launch");
    return -2;
  }
  auto lines = [](const float* p, long long ld) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0 ? 1 : 0; };
  const SgemmParams p{a, b, c, bias, M, N, K, slices, k_per, lda, ldb, ldc, lines(a, lda), lines(b, ldb), lines(c, ldc), relu, accumulate};
  return !a_rows ? launch<false, false>(p, tiles, stream) : b_rows ? launch<true, true>(p, tiles, stream) : launch<true, false>(p, tiles, stream);
}

// The derivative of a rectified layer at its output `out` [M, N] and the bias gradient in one pass; out null: the bias gradient alone.
KB_API int kb200_relu_bwd(const float* dy, const float* out, float* dz, float* db, int M, int N, int accumulate, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  relu_bwd_kernel<<<(unsigned)((N + 31) / 32), 256, 0, stream>>>(dy, out, dz, db, M, N, accumulate);
  KB_CHECK_LAUNCH("relu_bwd");
  return 0;
}

// Slices that kb200_sgemm_wgrad cuts K into: its workspace holds slices * (M + 1) * (N rounded up to 4) floats, 16-byte aligned.
KB_API int kb200_sgemm_wgrad_slices(int M, int N, int K) {
  int k_per;
  return M <= 0 || N <= 0 || K <= 0 ? 0 : wgrad_slices(M, N, K, &k_per);
}

// c [M, N] (+)= A^T B and db [N] (+)= B's column sums (db null: left out); A [K, M] and B [K, N] of row pitches lda and ldb, c contiguous.
KB_API int kb200_sgemm_wgrad(const float* a, const float* b, float* part, float* c, float* db, int M, int N, int K, long long lda, long long ldb, int add, int add_db,
                             cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || lda < M || ldb < N || ((uintptr_t)part & 15)) {
    kb200_set_error("sgemm_wgrad: an empty product, rows that overlap, or a workspace off its 16-byte line");
    return -2;
  }
  WgradParams p{a, b, part, M, N, K, 0, 0, 0, (N + 3) / 4 * 4, lda, ldb, 0, 0};
  p.slices = wgrad_slices(M, N, K, &p.k_per);
  auto lines = [](const float* q, long long ld, int cols) { return ((uintptr_t)q & 15) == 0 && ld % 4 == 0 && cols % 4 == 0 ? 1 : 0; };
  p.a_vec = lines(a, lda, M), p.b_vec = lines(b, ldb, N);
  const int wm = wgrad_rows(M);
  p.m_tiles = (M + wm - 1) / wm;
  const long long ctas = (long long)p.m_tiles * ((N + WN - 1) / WN) * p.slices, quads = (long long)(M + 1) * (p.pitch / 4);
  if (ctas > 0x7fffffffll || quads > 0x7fffff00ll) {
    kb200_set_error("sgemm_wgrad: too many tiles for one launch");
    return -2;
  }
  if (wm == 32)
    wgrad_kernel<32><<<(unsigned)ctas, 64, 0, stream>>>(p);
  else
    wgrad_kernel<64><<<(unsigned)ctas, 128, 0, stream>>>(p);
  KB_CHECK_LAUNCH("sgemm_wgrad");
  wgrad_sum_kernel<<<(unsigned)((quads + 31) / 32), 256, 0, stream>>>(part, c, db, M, N, p.pitch, p.slices, add, add_db);
  KB_CHECK_LAUNCH("sgemm_wgrad sums");
  return 0;
}
