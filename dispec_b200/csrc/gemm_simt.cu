// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) (+ residual[M,N]) on the 32-bit FMA units.
//
// This is the catch-all for sizes the tensor-core kernels refuse, and the product of floats of short
// rows (gemm_split.cu takes the others).  Every output element is
// one FMA chain over k = 0..K-1 in ascending order, so a row's result does not depend on
// which other rows are in the batch, nor on which of the kernels below computes it.
//
// Two kernels for floats, both fed by 16-byte asynchronous copies a few stages ahead, and one for bfloat16
// (`bf16_kernel`).  `few_rows_kernel` (up to 16 rows) streams W: it is bound by the bytes of W, or, where N is small, by the chain itself (K dependent FMAs of
// four cycles).  4 rows x 17,920 x 1,536: 44 us (210 with one 64 x 64 tile, single-float loads and no copies
// ahead); x 1,536 x 8,960: 62 us (1,056).
// `tile_kernel` holds BM x BN outputs in the registers of a block, 8 x 8 down to 4 x 2 a thread; it is bound
// by the issue of FMAs (the 128 x 128 tile: FMA pipe 64 % of its peak, issue slots 76 %) and, for the small
// tiles that few outputs need to reach all SMs, by shared-memory reads.  264 rows x 17,920 x 1,536: 381 us
// (38 TFLOP/s; 738 with that one tile); x 1,536 x 8,960: 275 us (1,026).
#include "common.cuh"

namespace {

template <typename TIn, typename TOut>
__device__ __forceinline__ void finish(float v, const TIn* bias, const TOut* residual, long ldr, TOut* C, long ldc,
                                       int m, int n) {
  if (bias) v += to_f32(bias[n]);
  if (residual) v += to_f32(residual[(size_t)m * ldr + n]);
  C[(size_t)m * ldc + n] = from_f32<TOut>(v);
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0));
}
template <int N>
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void end_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// ------------------------------------------------------------------ tiles of outputs in registers
constexpr int BK = 32, LDK = BK + 4;  // a row's 16-byte pieces start four banks behind its neighbour's

template <int BM, int BN>
constexpr int tile_stages() { return BM + BN > 192 ? 3 : 4; }
template <int BM, int BN>
constexpr int tile_smem() { return tile_stages<BM, BN>() * LDK * (BM + BN) * (int)sizeof(float); }

// COPY16: A and W have rows of whole 16-byte pieces, which are copied asynchronously.
template <int BM, int BN, int TM, int TN, bool COPY16>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
tile_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
            const float* __restrict__ residual, long ldr, float* __restrict__ C, long ldc, int M, int N, int K) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, STAGES = tile_stages<BM, BN>(), STAGE = LDK * (BM + BN);
  static_assert(TX % 8 == 0 && TY % 4 == 0 && THREADS % 32 == 0, "warps are 4 x 8 threads of the tile");
  extern __shared__ __align__(16) float tile_buf[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // a warp is 4 x 8 threads of the tile, every eight lanes in the same rows: a read of A has four addresses, one
  // for eight neighbouring lanes, which is much cheaper than four that alternate
  const int ty = (warp / (TX / 8)) * 4 + (lane >> 3);
  const int tx = (warp % (TX / 8)) * 8 + (lane & 7);
  // the tiles of a column block of W follow one another, so that W is read from memory once
  const int row_tiles = (M + BM - 1) / BM;
  const int m0 = (int)(blockIdx.x % row_tiles) * BM, n0 = (int)(blockIdx.x / row_tiles) * BN;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  auto fetch = [&](int stage, int k0) {
    float* to = tile_buf + stage * STAGE;
#pragma unroll 4
    for (int p = tid; p < (BM + BN) * (BK / 4); p += THREADS) {
      const int r = p / (BK / 4), k = k0 + p % (BK / 4) * 4;
      const bool is_a = r < BM;
      const int row = is_a ? m0 + r : n0 + r - BM;
      const bool inside = row < (is_a ? M : N);
      const float* src = is_a ? A + (size_t)row * lda + k : W + (size_t)row * K + k;
      float* dst = to + r * LDK + (k - k0);
      if constexpr (COPY16) {
        const bool there = inside && k < K;
        copy16(dst, there ? src : A, there);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e] = inside && k + e < K ? src[e] : 0.f;
      }
    }
  };
  const int steps = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) fetch(s, s * BK);
    end_group();
  }
  int stage = 0, next = STAGES - 1;
  for (int t = 0; t < steps; ++t) {
    wait_copies<STAGES - 2>();
    __syncthreads();  // the step's tiles are there for all, and all have left the stage that is filled next
    if (t + STAGES - 1 < steps) fetch(next, (t + STAGES - 1) * BK);
    end_group();
    const float* as = tile_buf + stage * STAGE + ty * LDK;
    const float* ws = tile_buf + stage * STAGE + (BM + tx) * LDK;
    // the operands of the next four k are read while those of these four are multiplied
    float4 a[2][TM], w[2][TN];
    auto read = [&](int to, int k) {
#pragma unroll
      for (int i = 0; i < TM; ++i) a[to][i] = *reinterpret_cast<const float4*>(as + i * TY * LDK + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[to][j] = *reinterpret_cast<const float4*>(ws + j * TX * LDK + k);
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      const int b = (k / 4) & 1;
      if (k + 4 < BK) read(b ^ 1, k + 4);
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[b][i].x, w[b][j].x, acc[i][j]);
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[b][i].y, w[b][j].y, acc[i][j]);
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[b][i].z, w[b][j].z, acc[i][j]);
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[b][i].w, w[b][j].w, acc[i][j]);
    }
    stage = stage + 1 == STAGES ? 0 : stage + 1;
    next = next + 1 == STAGES ? 0 : next + 1;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + i * TY + ty;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + j * TX + tx;
      if (n < N) finish(acc[i][j], bias, residual, ldr, C, ldc, m, n);
    }
  }
}

// ------------------------------------------------------------------ bfloat16 operands
// The sizes the tensor-core kernels refuse (a width that is no multiple of 8): single elements, turned to floats and
// stored k-major, 256 threads of 4 x 4 outputs.  Bound by the loads of single elements, which the many threads of a
// block cover best: 8 rows x 151,936 x 1,537 1,166 us, 64 rows x 1,536 x 1,537 205; in the row-major tiles above, 128
// threads of 8 x 4 outputs and stages that no asynchronous copy fills, 1,683 and 322.
constexpr int BF_M = 64, BF_N = 64, BF_K = 16, BF_T = 4;

template <typename TOut>
__global__ void __launch_bounds__(256)
bf16_kernel(const bf16* __restrict__ A, long lda, const bf16* __restrict__ W, const bf16* __restrict__ bias,
            const TOut* __restrict__ residual, long ldr, TOut* __restrict__ C, long ldc, int M, int N, int K) {
  __shared__ float as[BF_K][BF_M + 4];
  __shared__ float ws[BF_K][BF_N + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BF_M, n0 = blockIdx.x * BF_N;
  const int tx = tid % 16, ty = tid / 16;  // outputs rows ty * 4 .., columns tx * 4 ..
  float acc[BF_T][BF_T];
#pragma unroll
  for (int i = 0; i < BF_T; ++i)
#pragma unroll
    for (int j = 0; j < BF_T; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BF_K) {
#pragma unroll
    for (int e = 0; e < BF_M * BF_K / 256; ++e) {
      const int idx = tid + e * 256;
      const int r = idx / BF_K, c = idx % BF_K;
      const int m = m0 + r, n = n0 + r, k = k0 + c;
      as[c][r] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.f;
      ws[c][r] = (n < N && k < K) ? to_f32(W[(size_t)n * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BF_K; ++k) {
      float a[BF_T], w[BF_T];
#pragma unroll
      for (int i = 0; i < BF_T; ++i) a[i] = as[k][ty * BF_T + i];
#pragma unroll
      for (int j = 0; j < BF_T; ++j) w[j] = ws[k][tx * BF_T + j];
#pragma unroll
      for (int i = 0; i < BF_T; ++i)
#pragma unroll
        for (int j = 0; j < BF_T; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < BF_T; ++i) {
    const int m = m0 + ty * BF_T + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < BF_T; ++j) {
      const int n = n0 + tx * BF_T + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += to_f32(bias[n]);
      if (residual) v += to_f32(residual[(size_t)m * ldr + n]);
      C[(size_t)m * ldc + n] = from_f32<TOut>(v);
    }
  }
}

template <typename TOut>
int launch_bf16(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C, long ldc,
                int M, int N, int K, cudaStream_t stream) {
  bf16_kernel<TOut><<<dim3((N + BF_N - 1) / BF_N, (M + BF_M - 1) / BF_M), 256, 0, stream>>>(
      (const bf16*)A, lda, (const bf16*)W, (const bf16*)bias, (const TOut*)residual, ldr, (TOut*)C, ldc, M, N, K);
  DSP_CHECK_LAUNCH("dsp_gemm_simt");
  return 0;
}

// ------------------------------------------------------------------ up to 16 rows
constexpr int FEW_N = 16, FEW_K = 128, FEW_STAGES = 4, FEW_THREADS = 64;
constexpr int FEW_LD = FEW_K + 4;  // a row's 16-byte pieces start in another bank group than its neighbour's

// 16 columns and 4 MR rows a block; a thread owns one column of MR rows.  Rows of whole 16-byte pieces.
template <int MR>
__global__ void __launch_bounds__(FEW_THREADS)
few_rows_kernel(const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
                const float* __restrict__ residual, long ldr, float* __restrict__ C, long ldc, int M, int N, int K) {
  constexpr int ROWS = 4 * MR, STAGE = (FEW_N + ROWS) * FEW_LD;
  extern __shared__ __align__(16) float few_smem[];
  const int tid = threadIdx.x, n0 = blockIdx.x * FEW_N;
  const int nl = tid & 15, ml = tid >> 4;  // column, first row (rows ml, ml + 4, ...)
  auto fetch = [&](int s, int k0) {
    float* to = few_smem + s * STAGE;
#pragma unroll 4
    for (int i = tid; i < (FEW_N + ROWS) * (FEW_K / 4); i += FEW_THREADS) {
      const int r = i / (FEW_K / 4), k = k0 + (i % (FEW_K / 4)) * 4;
      const bool is_w = r < FEW_N;
      const int row = is_w ? n0 + r : r - FEW_N;
      const bool there = k < K && row < (is_w ? N : M);
      const float* src = is_w ? W + (size_t)row * K + k : A + (size_t)row * lda + k;
      copy16(to + r * FEW_LD + (k - k0), there ? src : A, there);
    }
  };
  const int steps = (K + FEW_K - 1) / FEW_K;
#pragma unroll
  for (int s = 0; s < FEW_STAGES - 1; ++s) {
    if (s < steps) fetch(s, s * FEW_K);
    end_group();
  }
  float acc[MR];
#pragma unroll
  for (int i = 0; i < MR; ++i) acc[i] = 0.f;
  for (int t = 0; t < steps; ++t) {
    wait_copies<FEW_STAGES - 2>();
    __syncthreads();
    if (t + FEW_STAGES - 1 < steps) fetch((t + FEW_STAGES - 1) % FEW_STAGES, (t + FEW_STAGES - 1) * FEW_K);
    end_group();
    const float* w = few_smem + (t % FEW_STAGES) * STAGE + nl * FEW_LD;
    const float* a = few_smem + (t % FEW_STAGES) * STAGE + (FEW_N + ml) * FEW_LD;
#pragma unroll 8
    for (int k = 0; k < FEW_K; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
      for (int i = 0; i < MR; ++i) {
        const float4 y = *reinterpret_cast<const float4*>(a + i * 4 * FEW_LD + k);
        acc[i] = fmaf(y.w, x.w, fmaf(y.z, x.z, fmaf(y.y, x.y, fmaf(y.x, x.x, acc[i]))));
      }
    }
  }
  const int n = n0 + nl;
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    const int m = ml + 4 * i;
    if (m < M && n < N) finish(acc[i], bias, residual, ldr, C, ldc, m, n);
  }
}

template <int BM, int BN, int TM, int TN, bool COPY16>
int launch_tile(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                long ldc, int M, int N, int K, cudaStream_t stream) {
  const long blocks = (long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  DSP_REQUIRE(blocks < (1l << 31), "dsp_gemm_simt: M=%d, N=%d too large for one launch", M, N);
  constexpr int smem = tile_smem<BM, BN>();
  auto* kernel = tile_kernel<BM, BN, TM, TN, COPY16>;
  DSP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kernel<<<(unsigned)blocks, (BM / TM) * (BN / TN), smem, stream>>>(
      (const float*)A, lda, (const float*)W, (const float*)bias, (const float*)residual, ldr, (float*)C, ldc, M, N, K);
  DSP_CHECK_LAUNCH("dsp_gemm_simt");
  return 0;
}

template <int MR>
int launch_few(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
               long ldc, int M, int N, int K, cudaStream_t stream) {
  constexpr int smem = FEW_STAGES * (FEW_N + 4 * MR) * FEW_LD * (int)sizeof(float);
  DSP_CUDA(cudaFuncSetAttribute(few_rows_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  few_rows_kernel<MR><<<(N + FEW_N - 1) / FEW_N, FEW_THREADS, smem, stream>>>(
      (const float*)A, lda, (const float*)W, (const float*)bias, (const float*)residual, ldr, (float*)C, ldc, M, N, K);
  DSP_CHECK_LAUNCH("dsp_gemm_simt");
  return 0;
}

// Cycles a block takes per k (measured at 1,965 MHz, K 8,960 and 1,536; aligned floats come with K below 1,536, the others
// with any): with an SM to itself, and its share of an
// SM that holds as many as fit.  The larger tiles need fewer shared-memory reads per product (128 x 128: 195 cycles
// of which 128 are the FMA units' own), the smaller ones reach more SMs when there are few outputs.
struct Tile {
  int bm, bn;
  float alone, shared;
};
constexpr Tile TILES[] = {{128, 128, 195.f, 195.f}, {96, 128, 165.f, 155.f}, {64, 128, 165.f, 108.f},
                          {96, 64, 94.f, 85.f},     {64, 64, 70.f, 57.f},    {96, 32, 61.f, 44.f},
                          {64, 32, 43.f, 29.f},     {32, 64, 44.f, 29.5f},   {32, 32, 30.f, 18.f}};
constexpr int NUM_TILES = sizeof(TILES) / sizeof(TILES[0]), FEW_TILE = NUM_TILES, FEW_MAX_ROWS = 16;

// The kernel whose busiest SM is done first.
int choose_tile(int M, int N) {
  const long sms = dsp_num_sms() > 0 ? dsp_num_sms() : 148;
  int best = 0;
  float least = 0.f;
  auto consider = [&](int i, long blocks, float alone, float shared) {
    const float cost = fmaxf(alone, (float)((blocks + sms - 1) / sms) * shared);
    if (i == 0 || cost < least) best = i, least = cost;
  };
  for (int i = 0; i < NUM_TILES; ++i)
    consider(i, (long)((M + TILES[i].bm - 1) / TILES[i].bm) * ((N + TILES[i].bn - 1) / TILES[i].bn), TILES[i].alone,
             TILES[i].shared);
  if (M <= FEW_MAX_ROWS)
    consider(FEW_TILE, (N + FEW_N - 1) / FEW_N, M <= 4 ? 13.2f : M <= 8 ? 18.4f : 23.8f, M <= 4 ? 4.1f : M <= 8 ? 6.1f : 9.8f);
  return best;
}
}  // namespace

// in_dtype: type of A, W and bias.  out_dtype: type of C and residual.  tile: -1 (by the rule above), an index
// into TILES, or their number for the kernel of few rows (comparisons; every one gives the same bits).
extern "C" int dsp_gemm_simt(const void* A, long lda, const void* W, const void* bias,
                             const void* residual, long ldr, void* C, long ldc, int M, int N, int K,
                             int in_dtype, int out_dtype, int tile, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  DSP_REQUIRE(K > 0, "dsp_gemm_simt: K=%d", K);
  DSP_REQUIRE(M <= 65535 * 64, "dsp_gemm_simt: M=%d too large for one launch", M);
  DSP_REQUIRE(tile >= -1 && tile <= FEW_TILE, "dsp_gemm_simt: no tile %d", tile);
#define DSP_TILE(...) \
  return launch_tile<__VA_ARGS__>(A, lda, W, bias, residual, ldr, C, ldc, M, N, K, stream)
#define DSP_FEW(MR) return launch_few<MR>(A, lda, W, bias, residual, ldr, C, ldc, M, N, K, stream)
  if (in_dtype == DSP_F32 && out_dtype == DSP_F32) {
    if (K % 4 || lda % 4 || (uintptr_t)A % 16 || (uintptr_t)W % 16) DSP_TILE(64, 64, 8, 4, false);
    DSP_REQUIRE(tile != FEW_TILE || M <= FEW_MAX_ROWS, "dsp_gemm_simt: %d rows are too many for the kernel of few rows", M);
    if (tile < 0) tile = choose_tile(M, N);
    switch (tile) {
      case 0: DSP_TILE(128, 128, 8, 8, true);
      case 1: DSP_TILE(96, 128, 12, 4, true);
      case 2: DSP_TILE(64, 128, 8, 8, true);
      case 3: DSP_TILE(96, 64, 12, 4, true);
      case 4: DSP_TILE(64, 64, 8, 4, true);
      case 5: DSP_TILE(96, 32, 6, 4, true);
      case 6: DSP_TILE(64, 32, 4, 4, true);
      case 7: DSP_TILE(32, 64, 4, 4, true);
      case 8: DSP_TILE(32, 32, 4, 2, true);
      default:
        if (M <= 4) DSP_FEW(1);
        if (M <= 8) DSP_FEW(2);
        DSP_FEW(4);
    }
  }
  if (in_dtype == DSP_BF16 && out_dtype == DSP_BF16) return launch_bf16<bf16>(A, lda, W, bias, residual, ldr, C, ldc, M, N, K, stream);
  if (in_dtype == DSP_BF16 && out_dtype == DSP_F32) return launch_bf16<float>(A, lda, W, bias, residual, ldr, C, ldc, M, N, K, stream);
#undef DSP_TILE
#undef DSP_FEW
  DSP_REQUIRE(false, "dsp_gemm_simt: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}
