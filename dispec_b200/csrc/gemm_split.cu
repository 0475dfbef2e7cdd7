// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) (+ residual[M,N]), floats in and out, on the fifth-generation tensor
// cores: the matrix product of the true 32-bit path.
//
// An operand times 2^24 is the sum of three bfloat16 values, x1 + x2 + x3 exactly (8 + 8 + 8 bits, each piece the rounded
// rest of the one before; the lowest bit of any float is 2^-149, so that no piece is smaller than the normal numbers), and
// of the nine products of pieces the six largest are formed: a1 w1, and a1 w2, a2 w1, a2 w2, a1 w3, a3 w1; what is left
// out is below 2^-24 of a product.  The a1 w1 of 128 k are summed in tensor memory, then added to 32-bit sums in registers (rounded to nearest, where the tensor cores cut sums off); the five
// small products, 2^-8 of them, are summed in tensor memory over all of K and added at the end.
//
// Roles are swapped as in gemm_stream.cu: 128 rows of W are the lanes, a chunk of up to 96 rows of A the columns.
//   warp 0       requests W and A (floats) by TMA, 32 k at a time, into a ring
//   warps 2..9   cut blocks into pieces, two groups of four warps in turn: W's go to tensor memory as the first
//                operand (a thread a row of W), A's to shared memory
//   warp 1       issues the products: 12 of K 16 for 32 k
//   warps 10..17 add the sums of 128 k to their registers, and finish the tile
// W's pieces in tensor memory keep them off the shared-memory port, which floats and A's pieces fill for some 880
// cycles for 32 k of 96 rows, beside 580 to 660 of the tensor cores.
//
// Against 64 bits, relative error of normal operands, this product and the chain of 32-bit FMAs (gemm_simt.cu): 1.3e-7
// and 7.0e-7 at K 1,536, 1.6e-7 and 1.7e-6 at K 8,960; operands of one sign, K 1,536, uniform 1.5e-7 and 5.9e-7, lognormal
// 6.7e-7 and 8.4e-7, squares 3.0e-7 and 6.0e-7.  us, the same two, launches one after the other: 264
// rows x 17,920 x 1,536 109 and 380, x 1,536 x 8,960 62 and 268, x 1,536 x 1,536 18 and 49; 4 rows x 17,920 x 1,536 26 and 37, x
// 1,536 x 8,960 40 and 57, x 151,936 x 1,536 162 and 204.
//
// What a result depends on: its row of A, its row of W, N and K.  K is split over a cluster by a rule on N and K
// alone, the pieces are summed in the same order for every width of a chunk, and so a row has the same bits alone and
// among others.
//
// Where the pieces do not hold, the result says so: an infinity or NaN among the operands, or one from 2^104 on, whose
// first piece is no bfloat16, gives NaN (x - x1 = -inf or NaN); sums from 2^76 on are not trusted, being near the end of
// the range of the scaled ones.  Such a result is formed again as one chain of 32-bit FMAs; so is one below 2^-60, whose
// bits are then those of gemm_simt.cu down to the subnormal numbers.
//
// Launched plainly, and every wait on an mbarrier is bounded; a wait that runs out is recorded in the device error word.
#include <cooperative_groups.h>

#include <atomic>

#include "tcgen05_common.cuh"

namespace cg = cooperative_groups;

namespace {
using namespace tc;
constexpr int ROWS_W = 128, BK = 32, UMMA_K = 16, CHUNK_KB = 4;  // blocks of k whose large products meet in tensor memory
constexpr int W_BYTES = ROWS_W * BK * 4;  // a block of W as floats, 128 bytes a row
constexpr int GROUPS = 2, GROUP_WARPS = 4, ADDERS = 8, FIRST_CONVERTER = 2, FIRST_ADDER = FIRST_CONVERTER + GROUPS * GROUP_WARPS;
constexpr int THREADS = 32 * (FIRST_ADDER + ADDERS);
constexpr int MAX_SPLITS = 8, MAX_ROWS = 96;
constexpr int STAGES = 4, W_COLS = 3 * BK / 2;  // blocks of k cut ahead; tensor-memory columns of a block's pieces of W

template <int NB> struct Cfg {
  // the pieces of two neighbouring blocks of A share rows of 128 bytes
  static constexpr int PIECE_BYTES = NB * 2 * BK * 2, PAIR_BYTES = 3 * PIECE_BYTES;
  static constexpr int RAW_BYTES = W_BYTES + NB * BK * 4;  // a block of W and of A as floats
  static constexpr int RAW_STAGES = NB <= 16 ? 11 : NB <= 32 ? 9 : NB <= 64 ? 7 : 5;
  static constexpr int SMEM = RAW_STAGES * RAW_BYTES + STAGES / 2 * PAIR_BYTES + 1024;
  // tensor memory: two sums of large products, one of small ones, the pieces of W
  static constexpr int W_AT = 3 * NB, USED = W_AT + STAGES * W_COLS, TMEM_COLS = USED <= 256 ? 256 : 512;
  static constexpr int MINE = NB / 2;           // columns of an adding thread
  static constexpr int ITEMS = (NB + 31) / 32;  // eight k of a row of A each, a converting thread's share of a block
  static_assert(USED <= 512 && SMEM <= 227 * 1024 - 512, "fits an SM");
  static_assert(NB * ROWS_W * 4 <= RAW_STAGES * RAW_BYTES, "the drained ring holds a tile");
};

struct Args {
  const float* A;
  long lda;
  const float* W;
  const float* bias;
  const float* residual;
  long ldr;
  float* C;
  long ldc;
  int M, N, K;
  int chunk_rows, chunks;  // rows of A a tile takes, tiles a block of W takes part in
  int kb_per_split;
  int a_wide;  // rows of A are whole 16-byte pieces
};

// of an operand, of a sum of products (two operands an instruction; without, the product is up to 2.5 % faster and the
// second and third pieces of operands below 2^-110 lose bits)
constexpr float SCALE = 0x1p24f, UNSCALE = 0x1p-48f;

// two floats times 2^24 as three pairs of bfloat16 values that add up to them
__device__ __forceinline__ void cut2(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  asm("{\n\t.reg .b64 t, s;\n\tmov.b64 t, {%0, %1};\n\tmov.b64 s, {%2, %2};\n\tmul.rn.f32x2 t, t, s;\n\tmov.b64 {%0, %1}, t;\n\t}"
      : "+f"(x), "+f"(y) : "f"(SCALE));
  p1 = pack2(x, y);
  x -= __uint_as_float(p1 << 16), y -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pack2(x, y);
  x -= __uint_as_float(p2 << 16), y -= __uint_as_float(p2 & 0xffff0000u);
  p3 = pack2(x, y);
}

template <int N> __device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]);
template <> __device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <> __device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// One result as one chain of 32-bit FMAs (K a multiple of 4, w on 16 bytes).  Sixteen operands of each side are on their
// way at a time, and a chain that is no number any more ends: rows that hold a NaN cost a few loads each.
__device__ __noinline__ float chain(const float* a, const float* w, int K) {
  float s = 0.f;
  int k = 0;
  for (; k + 16 <= K && s == s; k += 16) {
    float x[16];
    float4 y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(w + k + 4 * j);
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = a[k + j];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s = fmaf(x[4 * j], y[j].x, s), s = fmaf(x[4 * j + 1], y[j].y, s);
      s = fmaf(x[4 * j + 2], y[j].z, s), s = fmaf(x[4 * j + 3], y[j].w, s);
    }
  }
  for (; k < K && s == s; ++k) s = fmaf(a[k], w[k], s);
  return s;
}
__device__ __forceinline__ float finish(const Args& g, float v, int m, int n) {
  v *= UNSCALE;
  const float size = fabsf(v);
  if (!(size < 0x1p76f) || (size < 0x1p-60f && v != 0.f)) v = chain(g.A + (size_t)m * g.lda, g.W + (size_t)n * g.K, g.K);
  if (g.bias) v += g.bias[n];
  if (g.residual) v += g.residual[(size_t)m * g.ldr + n];
  return v;
}

template <int NB>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const Args g, int* err) {
  using C = Cfg<NB>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* pieces = smem + C::RAW_STAGES * C::RAW_BYTES;
  __shared__ __align__(8) uint64_t raw_full[C::RAW_STAGES], raw_empty[C::RAW_STAGES], ops_full[STAGES], ops_empty[STAGES],
      sum_full[2], sum_empty[2], small_full, small_empty;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = gridDim.y, kb_total = (g.K + BK - 1) / BK;
  const int kb0 = blockIdx.y * g.kb_per_split, num_kb = min(kb_total, kb0 + g.kb_per_split) - kb0;
  const int tiles = (g.N + ROWS_W - 1) / ROWS_W * g.chunks;  // (block of W, chunk of rows), chunks innermost

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::RAW_STAGES; ++s) mbar_init(&raw_full[s], 1), mbar_init(&raw_empty[s], GROUP_WARPS);
    for (int s = 0; s < STAGES; ++s) mbar_init(&ops_full[s], GROUP_WARPS), mbar_init(&ops_empty[s], 1);
    for (int b = 0; b < 2; ++b) mbar_init(&sum_full[b], 1), mbar_init(&sum_empty[b], ADDERS);
    mbar_init(&small_full, 1), mbar_init(&small_empty, ADDERS);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    const bool leader = elect_one();
    const uint64_t policy = g.chunks == 1 ? l2_policy_evict_first() : l2_policy_evict_normal();
    int s = 0, phase = 1;
    for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
      const int n0 = tile / g.chunks * ROWS_W, m0 = tile % g.chunks * g.chunk_rows;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&raw_empty[s], phase)) {
          failed = 1;
          break;
        }
        if (leader) {
          mbar_expect_tx(&raw_full[s], g.a_wide ? C::RAW_BYTES : W_BYTES);
          tma_load_2d_hint(smem + s * C::RAW_BYTES, &map_w, &raw_full[s], (kb0 + kb) * BK, n0, policy);
          if (g.a_wide) tma_load_2d(smem + s * C::RAW_BYTES + W_BYTES, &map_a, &raw_full[s], (kb0 + kb) * BK, m0);
        }
        if (++s == C::RAW_STAGES) s = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc(ROWS_W, NB);
    int it = 0, group = 0, local = 0;
    for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x, ++local) {
      bool ok = mbar_wait(&small_empty, (local & 1) ^ 1);
      for (int kb = 0; kb < num_kb && ok; ++kb, ++it) {
        const int buf = group & 1, p = it % STAGES;
        if (kb % CHUNK_KB == 0) ok = mbar_wait(&sum_empty[buf], ((group >> 1) & 1) ^ 1);
        ok = ok && mbar_wait(&ops_full[p], (it / STAGES) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t large = tmem + buf * NB, small = tmem + 2 * NB, w = tmem + C::W_AT + p * W_COLS;
        const uint64_t a = umma_desc(smem_u32(pieces + (p >> 1) * C::PAIR_BYTES)) + (p & 1) * 4;  // 64 bytes into the rows
        constexpr uint64_t PIECE = C::PIECE_BYTES >> 4;
        const bool last = kb % CHUNK_KB == CHUNK_KB - 1 || kb + 1 == num_kb;
        if (leader) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t a1 = a + k * 2, a2 = a1 + PIECE, a3 = a2 + PIECE;  // 32 bytes a step
            const uint32_t w1 = w + k * 8, w2 = w1 + BK / 2, w3 = w2 + BK / 2;
            umma_a_tmem(large, w1, a1, idesc, (kb % CHUNK_KB | k) != 0);
            umma_a_tmem(small, w1, a3, idesc, (kb | k) != 0);
            umma_a_tmem(small, w3, a1, idesc, 1);
            umma_a_tmem(small, w2, a2, idesc, 1);
            umma_a_tmem(small, w1, a2, idesc, 1);
            umma_a_tmem(small, w2, a1, idesc, 1);
          }
          umma_commit(&ops_empty[p]);
          if (last) umma_commit(&sum_full[buf]);
        }
        group += last;
      }
      if (!ok) {
        failed = 1;
        break;
      }
      if (leader) umma_commit(&small_full);
    }
  } else if (warp < FIRST_ADDER) {
    // ---- cutting operands into pieces: two groups of four warps, a thread a row of W, take the blocks in turn
    const int t = (threadIdx.x - 32 * FIRST_CONVERTER) & 127, mine = (warp - FIRST_CONVERTER) / GROUP_WARPS, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    // of A: rows a_row, a_row + 32, ...; k 8 (t & 3) and the seven after it (eight neighbouring lanes: rows 4 apart, so
    // that their stores meet no bank twice)
    const int a_row = (t >> 5) * 8 + ((t >> 2) & 1) * 4 + ((t >> 3) & 3);
    // the CTA's blocks are one sequence over its tiles: number `it` is block it % num_kb
    const int my_tiles = blockIdx.x < tiles ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int total = my_tiles * num_kb;
    for (int it = mine; it < total; it += GROUPS) {
      const int p = it % STAGES, s = it % C::RAW_STAGES;
      if (!__all_sync(0xffffffffu, mbar_wait(&raw_full[s], (it / C::RAW_STAGES) & 1))) {
        failed = 1;
        break;
      }
      const unsigned char* raw = smem + s * C::RAW_BYTES;
      uint32_t q[3][16];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 x = *reinterpret_cast<const float4*>(raw + row * 128 + ((c ^ (row & 7)) << 4));
        cut2(x.x, x.y, q[0][2 * c], q[1][2 * c], q[2][2 * c]);
        cut2(x.z, x.w, q[0][2 * c + 1], q[1][2 * c + 1], q[2][2 * c + 1]);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&ops_empty[p], ((it / STAGES) & 1) ^ 1))) {
        failed = 1;
        break;
      }
      tc_fence_after();
      const uint32_t to = tmem + C::W_AT + p * W_COLS + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
      for (int j = 0; j < 3; ++j) tmem_st16(to + j * (BK / 2), q[j]);
#pragma unroll
      for (int i = 0; i < C::ITEMS; ++i) {
        const int r = a_row + i * 32;
        if (r >= NB) break;
        float4 x[2];
        if (g.a_wide) {
#pragma unroll
          for (int e = 0; e < 2; ++e)
            x[e] = *reinterpret_cast<const float4*>(raw + W_BYTES + r * 128 + ((((t & 3) * 2 + e) ^ (r & 7)) << 4));
        } else {
          const int tile = (int)blockIdx.x + it / num_kb * (int)gridDim.x, k = (kb0 + it % num_kb) * BK + (t & 3) * 8;
          const int m = tile % g.chunks * g.chunk_rows + r;
          const float* src = g.A + (size_t)m * g.lda + k;
          const bool here = r < g.chunk_rows && m < g.M;
#pragma unroll
          for (int e = 0; e < 2; ++e)  // K is a multiple of 4
            x[e] = here && k + 4 * e < g.K ? make_float4(src[4 * e], src[4 * e + 1], src[4 * e + 2], src[4 * e + 3])
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        uint32_t u[3][4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          cut2(x[e].x, x[e].y, u[0][2 * e], u[1][2 * e], u[2][2 * e]);
          cut2(x[e].z, x[e].w, u[0][2 * e + 1], u[1][2 * e + 1], u[2][2 * e + 1]);
        }
        const uint32_t dst = smem_u32(pieces + (p >> 1) * C::PAIR_BYTES) + (r >> 3) * 1024 + (r & 7) * 128 +
                             ((((p & 1) * 4 + (t & 3)) ^ (r & 7)) << 4);
#pragma unroll
        for (int j = 0; j < 3; ++j) st_shared16(dst + j * C::PIECE_BYTES, make_uint4(u[j][0], u[j][1], u[j][2], u[j][3]));
      }
      tmem_st_wait();
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&raw_empty[s]), mbar_arrive(&ops_full[p]);
    }
  } else {
    // ---- adding up and finishing: a thread has one row of W, half of the chunk's rows
    const int quarter = warp & 3, half = (warp - FIRST_ADDER) >> 2, row = quarter * 32 + lane;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    constexpr int STEP = C::MINE < 16 ? 8 : 16;
    int group = 0, local = 0;
    for (int tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x, ++local) {
      float sum[C::MINE];
#pragma unroll
      for (int c = 0; c < C::MINE; ++c) sum[c] = 0.f;
      auto add = [&](uint32_t from) {
#pragma unroll
        for (int c = 0; c < C::MINE; c += STEP) {
          uint32_t v[STEP];
          tmem_ld<STEP>(tmem + lanes + from + half * C::MINE + c, v);
#pragma unroll
          for (int j = 0; j < STEP; ++j) sum[c + j] += __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
      };
      bool ok = true;
      for (int kb = 0; kb < num_kb && ok; kb += CHUNK_KB, ++group) {
        const int buf = group & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&sum_full[buf], (group >> 1) & 1));
        if (!ok) break;
        tc_fence_after();
        add(buf * NB);
        if (lane == 0) mbar_arrive(&sum_empty[buf]);
      }
      ok = ok && __all_sync(0xffffffffu, mbar_wait(&small_full, local & 1));
      if (!ok) {
        failed = 1;
        break;
      }
      tc_fence_after();
      add(2 * NB);
      if (lane == 0) mbar_arrive(&small_empty);
      const int m0 = tile % g.chunks * g.chunk_rows, rows = min(g.chunk_rows, g.M - m0), n = tile / g.chunks * ROWS_W + row;
      if (splits == 1) {
#pragma unroll
        for (int c = 0; c < C::MINE; ++c) {
          const int m = half * C::MINE + c;
          if (m < rows && n < g.N) g.C[(size_t)(m0 + m) * g.ldc + n] = finish(g, sum[c], m0 + m, n);
        }
      } else {  // every product has run: the ring is free
        float* part = reinterpret_cast<float*>(smem);  // [row of A][128]
#pragma unroll
        for (int c = 0; c < C::MINE; ++c) part[(half * C::MINE + c) * ROWS_W + row] = sum[c];
      }
    }
  }

  if (splits > 1) {
    // one tile a CTA; the cluster's CTAs finish the rows of A in turn, adding the parts in rank order
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();
    cluster.sync();
    const int rank = (int)cluster.block_rank(), tile = blockIdx.x;
    const int m0 = tile % g.chunks * g.chunk_rows, rows = min(g.chunk_rows, g.M - m0);
    const float* part = reinterpret_cast<const float*>(smem);
    for (int i = threadIdx.x; !failed; i += THREADS) {
      const int m = i / ROWS_W * splits + rank, n = tile / g.chunks * ROWS_W + i % ROWS_W;
      if (m >= rows) break;
      float v[MAX_SPLITS];
#pragma unroll
      for (int r = 0; r < MAX_SPLITS; ++r) v[r] = r < splits ? cluster.map_shared_rank(part, r)[m * ROWS_W + i % ROWS_W] : 0.f;
      float total = v[0];
#pragma unroll
      for (int r = 1; r < MAX_SPLITS; ++r)
        if (r < splits) total += v[r];
      if (n < g.N) g.C[(size_t)(m0 + m) * g.ldc + n] = finish(g, total, m0 + m, n);
    }
    __syncthreads();
    cluster.sync();  // nobody reads this CTA's part any more
  }
  tc_fence_before();
  __syncthreads();
  if (failed) {
    if (threadIdx.x == 0) atomicOr(err, DSP_ERR_WAIT_LIMIT);
    for (int i = 0; i < 2000; ++i) __nanosleep(100);  // copies that are still on their way land
  }
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
}

template <int NB>
int launch(const CUtensorMap& map_w, const Args& g, int tiles, int splits, int sms, int* err, cudaStream_t stream) {
  auto kernel = gemm_split_kernel<NB>;
  CUtensorMap map_a = map_w;  // not used where A's rows are no whole pieces
  DSP_REQUIRE(!g.a_wide || make_map_f32(&map_a, g.A, g.M, g.K, g.lda, NB), "dsp_gemm_split: cannot encode the tensor map of A");
  static std::atomic<bool> configured[MAX_DEVICES] = {};
  const int device = current_device();
  DSP_REQUIRE(device >= 0, "dsp_gemm_split: the current device is not known");
  if (!configured[device].load(std::memory_order_relaxed)) {
    DSP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<NB>::SMEM));
    DSP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    configured[device].store(true, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits > 1 || tiles < sms ? tiles : sms, splits, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = Cfg<NB>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = splits;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  DSP_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_w, map_a, g, err));
  return 0;
}
}  // namespace

// W: rows of whole 16-byte pieces (K a multiple of 4, the pointer 16-byte aligned); A: any address and row stride.
extern "C" int dsp_gemm_split(const float* A, long lda, const float* W, const float* bias, const float* residual, long ldr,
                              float* C, long ldc, int M, int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  DSP_REQUIRE(K > 0 && K % 4 == 0 && ((uintptr_t)W & 15) == 0, "dsp_gemm_split: K=%d must be a multiple of 4 and W 16-byte aligned", K);
  int* err = dsp_device_error_ptr();
  DSP_REQUIRE(err != nullptr, "dsp_gemm_split: no device error word");
  const int sms = dsp_num_sms() > 0 ? dsp_num_sms() : 148;
  CUtensorMap map_w;
  DSP_REQUIRE(make_map_f32(&map_w, W, N, K, K, ROWS_W), "dsp_gemm_split: cannot encode the tensor map of W");
  Args g = {A, lda, W, bias, residual, ldr, C, ldc, M, N, K};
  g.chunks = (M + MAX_ROWS - 1) / MAX_ROWS;
  g.chunk_rows = (M + g.chunks - 1) / g.chunks;
  g.chunks = (M + g.chunk_rows - 1) / g.chunk_rows;
  g.a_wide = lda % 4 == 0 && lda >= K && ((uintptr_t)A & 15) == 0;  // (rows that overlap are no tensor map's)
  // K is split where there are few blocks of W, by their number alone: a row's sums must not depend on how many rows
  // there are.  Up to 14 blocks as many times as leaves clusters that fit beside one another with three chunks of rows
  // (36 clusters of four do not); from there on with one chunk (33 clusters of four, 45 of three, 74 of two): not
  // split from 23 blocks on and in two parts below, one row x 3,072 x 2,048 took 26.9 us, in four 11.6 (chain of FMAs 15.6),
  // x 2,048 x 1,536 13.8 and 10.0 (10.9), x 8,960 x 3,072 39.7 and about 26 in two (31.9); 264 rows x 3,072 x 2,048 45 and 49 (103),
  // x 2,048 x 1,536 23 and 29 (62).  Where it is still behind the chain: up to 4 rows x 9,300 to 12,000 and 19,000 to 24,000, at
  // most 23.2 us for 18.5.
  const int blocks = (N + ROWS_W - 1) / ROWS_W, kb_total = (K + BK - 1) / BK;
  int splits = blocks <= 14 ? 44 / blocks : blocks <= 32 ? 4 : blocks <= 44 ? 3 : blocks <= 72 ? 2 : 1;
  if (splits > MAX_SPLITS) splits = MAX_SPLITS;
  if (splits > kb_total / 8) splits = kb_total / 8;
  if (splits < 1) splits = 1;
  g.kb_per_split = (kb_total + splits - 1) / splits;
  splits = (kb_total + g.kb_per_split - 1) / g.kb_per_split;
  const long tiles = (long)blocks * g.chunks;
  DSP_REQUIRE(tiles < (1l << 31), "dsp_gemm_split: M=%d, N=%d too large for one launch", M, N);
  if (g.chunk_rows <= 16) return launch<16>(map_w, g, (int)tiles, splits, sms, err, stream);
  if (g.chunk_rows <= 32) return launch<32>(map_w, g, (int)tiles, splits, sms, err, stream);
  if (g.chunk_rows <= 64) return launch<64>(map_w, g, (int)tiles, splits, sms, err, stream);
  return launch<96>(map_w, g, (int)tiles, splits, sms, err, stream);
}
