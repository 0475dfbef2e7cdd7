// Attention over a cached latent for portions of prompts, on the fifth-generation tensor cores.
//
// The kernel in attn_latent.cu works on the latents themselves (scores over 512 + 64 numbers, sums over 512, for
// every head), which costs 2,176 operations a query, key and head but needs no memory: right for single tokens,
// whose time is the reading of the cache.  A portion of a prompt pays 3.4 times the operations of keys and
// values of 128 + 64 and 128, on mma.sync.  Here the latents of the portion's keys are gathered from the pages
// (latent_gather_kernel), one ordinary product expands them to every head's keys and values, rows
// [key of head 0 | key of head 1 | ... | value of head 0 | ...], and this kernel runs over those rows.
//
// A tile is 128 tokens of one sequence and one head.  Roles as in attn_tcgen05.cu, one CTA per tile:
//   warp 0      requests the K tiles (64 keys: the expanded part and the rotated part all heads share)
//   warp 12     requests the V tiles
//   warps 1, 11 one thread each issues S[i] = Q K[i]^T for one softmax group
//   warp 10     one thread issues O[i % 2] += P[i] V[i]
//   warps 2..9  two softmax groups of four warps, group g the key tiles g, g + 2, ...; thread r owns row r.
// Tensor memory (512 columns): two score buffers of 64, two outputs of DV, P of both groups, and the unrotated
// part of Q as the A operand; Q's rotated part (turned here, in 32-bit, and rounded) is an A operand in shared
// memory, because with it the tensor memory would need 544 columns.
// Every wait on a barrier is bounded; a wait that runs out sets the device error word and the CTA returns after
// freeing its tensor memory.
//
// 2,500 tokens in two prompts (833 and 1,667), 12 heads of 128 (+ 64) on latents of 512: 49 us, with 11 for the
// gathering and 19 for the expanding product, in place of 481 in the kernel on the latents and 79 for its two products
// by head; the whole step of eight layers, four of them of this kind, 5.98 -> 4.06 ms.  A key tile takes about 1,300
// cycles (a chain of waits: scores, exponentials, P, output), of which the tensor pipe is busy 640.
#include "tcgen05_common.cuh"

#if !defined(DSP_DK) || !defined(DSP_DV)
#error "compile with -DDSP_DK=<unrotated key size> -DDSP_DV=<value size>"
#endif

namespace {
using namespace tc;

constexpr int DK = DSP_DK, DV = DSP_DV, DR = 64;  // key parts (unrotated, rotated) and values of a head
static_assert((DK == 64 || DK == 128) && (DV == 64 || DV == 128), "this kernel is built for heads of 64 and 128");
constexpr int BM = 128, BN = 64, THREADS = 13 * 32;
constexpr int PV_WARP = 10, S1_WARP = 11, V_WARP = 12;
constexpr int SLICE = BN * 128;  // bytes of 64 keys x 64 columns
constexpr int K_BYTES = (DK / 64 + 1) * SLICE, V_BYTES = DV / 64 * SLICE, QR_BYTES = BM * 128;
constexpr int K_STAGES = 4, V_STAGES = 6;
constexpr int SMEM_BYTES = QR_BYTES + K_STAGES * K_BYTES + V_STAGES * V_BYTES + 1024;
static_assert(SMEM_BYTES + 2048 <= 227 * 1024, "dynamic and static shared memory of a CTA");
constexpr int S_COLS = BN, O_COL = 2 * S_COLS, P_COLS = BN / 2, P_COL = O_COL + 2 * DV, Q_COL = P_COL + 2 * P_COLS;
constexpr int TMEM_COLS = 512;
static_assert(Q_COL + DK / 2 <= TMEM_COLS, "tensor memory layout");
constexpr float RESCALE_STEP = 8.f;  // the running maximum follows the true one in steps of 2^8

struct Params {
  const bf16* q;
  long q_stride;
  int q_head_stride, qr_off;  // head h's columns start at h * q_head_stride, its part to be rotated qr_off further
  const float* inv_freq;
  int rot, layout;
  float mag;
  const int *q_start, *ctx_len, *tile_seq, *tile_tok0;
  int tile_offset, singles, window;
  const unsigned long long* bad;  // [portion][max_tiles] keys (of 64) whose page could not be read
  int max_tiles;
  bf16* out;
  long out_stride;
  const float* gate;
  long ldg;
  const float* sink;
  float scale_log2;
  int* err;
};

// Keys of a portion's sequence that are expanded: [first, ctx), first a multiple of 64.
__device__ __forceinline__ int first_key(int ctx, int q_len, int window) {
  return window > 0 ? max(0, ctx - q_len - window + 1) / BN * BN : 0;
}
// Row of the expanded keys at which sequence `seq` begins: portions one after the other, in the batch's order.
__device__ __forceinline__ int first_row(const int* q_start, const int* ctx_len, int singles, int seq, int window) {
  int sum = 0;
  for (int s = singles + (int)(threadIdx.x & 31); s < seq; s += 32)
    sum += ctx_len[s] - first_key(ctx_len[s], q_start[s + 1] - q_start[s], window);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

__global__ void __launch_bounds__(THREADS, 1)
attn_latent_prompt_kernel(const Params p, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_v) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);  // swizzle atoms are 1024 bytes
  __shared__ __align__(8) uint64_t k_full[K_STAGES], k_empty[K_STAGES], v_full[V_STAGES], v_empty[V_STAGES];
  __shared__ __align__(8) uint64_t s_full[2], s_free[2], p_full[2], o_done[2], q_ready;
  __shared__ float merge_m[BM], merge_l[BM];
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // later tiles of a prompt see more keys: the longest work of all heads is scheduled first
  const int head = blockIdx.x, tile = ((int)gridDim.y - 1 - (int)blockIdx.y) + p.tile_offset, H = gridDim.x;
  const int seq = p.tile_seq[tile], tok0 = p.tile_tok0[tile];
  const int qs = p.q_start[seq], q_len = p.q_start[seq + 1] - qs, ctx = p.ctx_len[seq];
  if (ctx <= 0 || q_len <= 0 || tok0 >= q_len) return;
  const int nrows = min(BM, q_len - tok0);
  const int pos0 = ctx - q_len + tok0, pos_last = pos0 + nrows - 1;
  const int lo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;          // first key any row sees
  const int lo_top = p.window > 0 ? max(0, pos_last - p.window + 1) : 0;  // first key every row sees
  const int kt_begin = lo / BN, n_kt = pos_last / BN + 1 - kt_begin;
  const int first = first_key(ctx, q_len, p.window);
  const int row0 = first_row(p.q_start, p.ctx_len, p.singles, seq, p.window) - first;  // + key: its expanded row
  const unsigned long long* bad_of = p.bad + (size_t)(seq - p.singles) * p.max_tiles - first / BN;  // [key tile]

  unsigned char* qr_s = smem;                       // [128 rows][128 bytes]
  unsigned char* k_s = qr_s + QR_BYTES;             // [stage][slice][64 keys][128 bytes], the rotated part last
  unsigned char* v_s = k_s + K_STAGES * K_BYTES;

  if (tid == 0) {
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < V_STAGES; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&s_free[b], 4);
      mbar_init(&p_full[b], 4);
      mbar_init(&o_done[b], 1);
    }
    mbar_init(&q_ready, 8);  // four warps write the unrotated part, four the rotated one
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  if (warp >= 2 && warp < 6) {
    // Q, unrotated part: thread r writes row r to lane r of the tensor memory, two bfloat16 per column
    const int r = (warp & 3) * 32 + lane;
    const uint4* src = reinterpret_cast<const uint4*>(p.q + (size_t)(qs + tok0 + min(r, nrows - 1)) * p.q_stride +
                                                      (size_t)head * p.q_head_stride);
    const uint32_t q_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)Q_COL;
#pragma unroll
    for (int c0 = 0; c0 < DK / 2; c0 += 32) {
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 v = r < nrows ? __ldg(src + c0 / 4 + c) : make_uint4(0, 0, 0, 0);
        w[4 * c] = v.x, w[4 * c + 1] = v.y, w[4 * c + 2] = v.z, w[4 * c + 3] = v.w;
      }
      tmem_st32(q_addr + (uint32_t)c0, w);
    }
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_ready);
  } else if (warp >= 6 && warp < 10) {
    // Q, the part to be rotated: thread r turns row r in 32-bit and writes it, rounded, as a swizzled row of 128 bytes
    const int r = (warp & 3) * 32 + lane;
    const uint4* src = reinterpret_cast<const uint4*>(p.q + (size_t)(qs + tok0 + min(r, nrows - 1)) * p.q_stride +
                                                      (size_t)head * p.q_head_stride + p.qr_off);
    uint4 raw[8];
    bf16* x = reinterpret_cast<bf16*>(raw);
#pragma unroll
    for (int c = 0; c < 8; ++c) raw[c] = r < nrows ? __ldg(src + c) : make_uint4(0, 0, 0, 0);
    const int half = p.rot / 2;
    const float pos = (float)(pos0 + r);
    if (p.layout == 0) {
#pragma unroll
      for (int i = 0; i < DR / 2; ++i) {
        if (i < half) {
          float sn, cs;
          sincosf(pos * p.inv_freq[i], &sn, &cs);
          sn *= p.mag, cs *= p.mag;
          const float u = __bfloat162float(x[2 * i]), v = __bfloat162float(x[2 * i + 1]);
          x[2 * i] = __float2bfloat16(u * cs - v * sn);
          x[2 * i + 1] = __float2bfloat16(v * cs + u * sn);
        }
      }
    } else {
      for (int i = 0; i < half; ++i) {
        float sn, cs;
        sincosf(pos * p.inv_freq[i], &sn, &cs);
        sn *= p.mag, cs *= p.mag;
        const float u = __bfloat162float(x[i]), v = __bfloat162float(x[i + half]);
        x[i] = __float2bfloat16(u * cs - v * sn);
        x[i + half] = __float2bfloat16(v * cs + u * sn);
      }
    }
    const uint32_t dst = smem_u32(qr_s) + (uint32_t)r * 128u;
#pragma unroll
    for (int c = 0; c < 8; ++c) st_shared16(dst + (uint32_t)((c ^ (r & 7)) * 16), raw[c]);
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_ready);
  }

  if (warp == 0) {
    const bool leader = elect_one();
    for (int i = 0; i < n_kt; ++i) {
      const int s = i % K_STAGES;
      if (!mbar_wait(&k_empty[s], ((i / K_STAGES) & 1) ^ 1)) {
        failed = 1;
        break;
      }
      const int row = row0 + (kt_begin + i) * BN;
      if (leader) {
        mbar_expect_tx(&k_full[s], K_BYTES);
        tma_load_3d(k_s + s * K_BYTES, &map_k, &k_full[s], 0, row, head * (DK / 64));
        tma_load_2d(k_s + s * K_BYTES + DK / 64 * SLICE, &map_r, &k_full[s], 0, row);
      }
    }
  } else if (warp == V_WARP) {
    const bool leader = elect_one();
    for (int i = 0; i < n_kt; ++i) {
      const int s = i % V_STAGES;
      if (!mbar_wait(&v_empty[s], ((i / V_STAGES) & 1) ^ 1)) {
        failed = 1;
        break;
      }
      if (leader) {
        mbar_expect_tx(&v_full[s], V_BYTES);
        tma_load_3d(v_s + s * V_BYTES, &map_v, &v_full[s], 0, row0 + (kt_begin + i) * BN, H * (DK / 64) + head * (DV / 64));
      }
    }
  } else if (warp == 1 || warp == S1_WARP) {
    {
      const bool leader = elect_one();
      const uint32_t idesc_s = umma_idesc(BM, BN);
      const uint64_t k_desc0 = umma_desc(smem_u32(k_s)), qr_desc = umma_desc(smem_u32(qr_s));
      bool ok = mbar_wait(&q_ready, 0);
      tc_fence_after();
      for (int a = warp == 1 ? 0 : 1; a < n_kt && ok; a += 2) {
        const int s = a % K_STAGES;
        ok = a < 2 ? mbar_wait(&k_full[s], (a / K_STAGES) & 1)
                   : mbar_wait_both(&k_full[s], (a / K_STAGES) & 1, &s_free[a & 1], ((a - 2) >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint64_t k_desc = k_desc0 + (uint64_t)(s * (K_BYTES >> 4));
        const uint32_t tmem_s = tmem_base + (uint32_t)((a & 1) * S_COLS);
        if (leader) {
#pragma unroll
          for (int k = 0; k < DK / 16; ++k)
            umma_a_tmem(tmem_s, tmem_base + (uint32_t)(Q_COL + k * 8),
                        k_desc + (uint64_t)(((k >> 2) * SLICE + (k & 3) * 32) >> 4), idesc_s, k != 0);
#pragma unroll
          for (int k = 0; k < DR / 16; ++k)
            umma(tmem_s, qr_desc + (uint64_t)(k * 2), k_desc + (uint64_t)((DK / 64 * SLICE + k * 32) >> 4), idesc_s, 1);
          umma_commit(&s_full[a & 1]);
          umma_commit(&k_empty[s]);
        }
      }
      if (!ok) failed = 1;
    }
  } else if (warp == PV_WARP) {
    {
      const bool leader = elect_one();
      const uint32_t idesc_o = umma_idesc(BM, DV) | (1u << 16);  // B (values) is N-major
      const uint64_t v_desc0 = umma_desc_mn(smem_u32(v_s), SLICE);
      bool ok = true;
      for (int b = 0; b < n_kt && ok; ++b) {
        const int g = b & 1, st = b % V_STAGES;
        ok = mbar_wait_both(&v_full[st], (b / V_STAGES) & 1, &p_full[g], (b >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint64_t v_desc = v_desc0 + (uint64_t)(st * (V_BYTES >> 4));
        if (leader) {
#pragma unroll
          for (int k = 0; k < BN / 16; ++k)
            umma_a_tmem(tmem_base + (uint32_t)(O_COL + g * DV), tmem_base + (uint32_t)(P_COL + g * P_COLS + k * 8),
                        v_desc + (uint64_t)(k * 128), idesc_o, (b >= 2) || k != 0);
          umma_commit(&v_empty[st]);
          umma_commit(&o_done[g]);
        }
      }
      if (!ok) failed = 1;
    }
  } else {
    // ---- softmax groups: thread r of group g owns row r for the key tiles g, g + 2, ...
    const int g = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const bool row_ok = r < nrows;
    const int pos_r = pos0 + r, lo_r = p.window > 0 ? pos_r - p.window + 1 : 0;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + (uint32_t)(g * S_COLS), o_addr = lane_addr + (uint32_t)(O_COL + g * DV);
    const uint32_t p_addr = lane_addr + (uint32_t)(P_COL + g * P_COLS);
    const float scale = p.scale_log2;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    int j = 0;  // tiles of this group so far
    unsigned long long bad_next = g < n_kt ? bad_of[kt_begin + g] : 0ull;
    for (int i = g; i < n_kt; i += 2, ++j) {
      const int key0 = (kt_begin + i) * BN;
      const unsigned long long bad = bad_next;
      if (i + 2 < n_kt) bad_next = bad_of[kt_begin + i + 2];
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full[g], j & 1))) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sv[64];
      {
        uint32_t a[32], b[32];
        tmem_ld32_nowait(s_addr, a);
        tmem_ld32_nowait(s_addr + 32, b);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          sv[c] = a[c];
          sv[32 + c] = b[c];
        }
      }
      // the scores are in registers: the next scores of this group may overwrite S[g]
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[g]);
      // tiles every row of the CTA sees whole (most of them) skip the mask
      if (!(key0 + BN - 1 <= pos0 && key0 >= lo_top) || bad != 0ull) {
#pragma unroll
        for (int c = 0; c < 64; ++c) {
          const int key = key0 + c;
          const bool vis = row_ok && key <= pos_r && key >= lo_r && !((bad >> c) & 1ull);
          sv[c] = vis ? sv[c] : 0xff800000u;  // -inf
        }
      }
      float t0 = -INFINITY, t1 = -INFINITY, t2 = -INFINITY, t3 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 64; c += 4) {
        t0 = fmaxf(t0, __uint_as_float(sv[c]));
        t1 = fmaxf(t1, __uint_as_float(sv[c + 1]));
        t2 = fmaxf(t2, __uint_as_float(sv[c + 2]));
        t3 = fmaxf(t3, __uint_as_float(sv[c + 3]));
      }
      const float tmax = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)) * scale;  // the scale is positive
      // the running maximum moves only when the true one is more than 2^8 ahead: P stays below 2^8
      const float m_new = (tmax > m_run + RESCALE_STEP || m_run == -INFINITY) ? fmaxf(tmax, m_run) : m_run;
      const float alpha = m_new == m_run ? 1.f : ex2(m_run - m_new);  // 0 on a row's first visible tile
      m_run = m_new;
      const float neg_m = m_new == -INFINITY ? 0.f : -m_new;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 64; c += 4) {
        const float e0 = ex2(fmaf(__uint_as_float(sv[c]), scale, neg_m));
        const float e1 = ex2(fmaf(__uint_as_float(sv[c + 1]), scale, neg_m));
        const float e2 = ex2(fmaf(__uint_as_float(sv[c + 2]), scale, neg_m));
        const float e3 = ex2(fmaf(__uint_as_float(sv[c + 3]), scale, neg_m));
        a0 += e0;
        a1 += e1;
        a2 += e2;
        a3 += e3;
        pk[c / 2] = pack2(e0, e1);
        pk[c / 2 + 1] = pack2(e2, e3);
      }
      l_run = l_run * alpha + ((a0 + a1) + (a2 + a3));
      // the group's previous O[g] += P V must be complete before O[g] is rescaled and P[g] rewritten
      if (j > 0) {
        if (!__all_sync(0xffffffffu, mbar_wait(&o_done[g], (j - 1) & 1))) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
          for (int c0 = 0; c0 < DV; c0 += 32) {
            uint32_t ov[32];
            tmem_ld32(o_addr + (uint32_t)c0, ov);
#pragma unroll
            for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * alpha);
            tmem_st32(o_addr + (uint32_t)c0, ov);
          }
          tmem_st_wait();
        }
      }
      tmem_st32(p_addr, pk);  // P row r: 64 bfloat16 in the 32 columns of the group's A operand
      // value rows that no row of this tile may see are zeroed: 0 times what lies there could be no number
      if (key0 < lo || key0 + BN - 1 > pos_last || bad != 0ull) {
        if (!__all_sync(0xffffffffu, mbar_wait(&v_full[i % V_STAGES], (i / V_STAGES) & 1))) {
          ok = false;
          break;
        }
        const int key_row = r >> 1, key = key0 + key_row;  // two threads per key row
        if (key > pos_last || key < lo || ((bad >> key_row) & 1ull)) {
          const uint32_t row_addr = smem_u32(v_s + (i % V_STAGES) * V_BYTES) + (uint32_t)key_row * 128u +
                                    (uint32_t)(r & 1) * 64u;
#pragma unroll
          for (int h = 0; h < DV / 64; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c) st_shared16(row_addr + h * SLICE + c * 16, make_uint4(0, 0, 0, 0));
        }
        fence_async_smem();
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[g]);
    }
    // the group's last product
    if (ok && j > 0 && !__all_sync(0xffffffffu, mbar_wait(&o_done[g], (j - 1) & 1))) ok = false;
    if (!ok) failed = 1;
    if (g == 1) {
      merge_m[r] = m_run;
      merge_l[r] = l_run;
    }
    tc_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");  // the eight softmax warps
    if (g == 0 && !failed) {
      // ---- merge the two groups' partial results (two key splits) and the sink, and store row r
      tc_fence_after();
      const bool two = n_kt > 1;  // group 1 had tiles: O[1] holds its part
      const float m1 = two ? merge_m[r] : -INFINITY, l1 = two ? merge_l[r] : 0.f;
      const float z = p.sink ? p.sink[head] * 1.4426950408889634f : -INFINITY;
      const float M = fmaxf(fmaxf(m_run, m1), z);
      const float w0 = m_run == -INFINITY ? 0.f : ex2(m_run - M);
      const float w1 = m1 == -INFINITY ? 0.f : ex2(m1 - M);
      const float denom = l_run * w0 + l1 * w1 + (z == -INFINITY ? 0.f : ex2(z - M));
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
      const float f0 = w0 * inv, f1 = w1 * inv;
      const size_t row = (size_t)(qs + tok0 + r), col = (size_t)head * DV;
      bf16* dst = p.out + (row_ok ? row * p.out_stride + col : 0);
      const float* gate = p.gate && row_ok ? p.gate + row * p.ldg + col : nullptr;
      // every lane takes part in the warp-wide loads of tensor memory; lanes without a row store nothing
#pragma unroll 1
      for (int c0 = 0; c0 < DV; c0 += 32) {
        uint32_t ov[32];
        tmem_ld32(lane_addr + (uint32_t)(O_COL + c0), ov);
        if (two) {
          uint32_t ow[32];
          tmem_ld32(lane_addr + (uint32_t)(O_COL + DV + c0), ow);
#pragma unroll
          for (int c = 0; c < 32; ++c)
            ov[c] = __float_as_uint(__uint_as_float(ov[c]) * f0 + __uint_as_float(ow[c]) * f1);
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * f0);
        }
        if (row_ok) {
          if (gate) {
#pragma unroll
            for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) / (1.f + expf(-gate[c0 + c])));
          }
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 w;
            w.x = pack2(__uint_as_float(ov[c]), __uint_as_float(ov[c + 1]));
            w.y = pack2(__uint_as_float(ov[c + 2]), __uint_as_float(ov[c + 3]));
            w.z = pack2(__uint_as_float(ov[c + 4]), __uint_as_float(ov[c + 5]));
            w.w = pack2(__uint_as_float(ov[c + 6]), __uint_as_float(ov[c + 7]));
            *reinterpret_cast<uint4*>(dst + c0 + c) = w;
          }
        }
        __syncwarp();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (failed) {
    if (threadIdx.x == 0) atomicOr(p.err, DSP_ERR_WAIT_LIMIT);
    // let copies that are still on their way land before the shared memory goes away
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// One block per (64 keys, portion): copies the keys' latents and rotated parts from the pages to rows that follow
// one another, and notes which keys' pages could not be read.  R, r: multiples of 8.
constexpr int GATHER_THREADS = 256;
__global__ void __launch_bounds__(GATHER_THREADS)
latent_gather_kernel(const bf16* __restrict__ c_pool, const bf16* __restrict__ r_pool, const int* __restrict__ page_table,
                     int pt_stride, const int* __restrict__ q_start, const int* __restrict__ ctx_len, int singles,
                     int window, bf16* __restrict__ c_rows, bf16* __restrict__ r_rows,
                     unsigned long long* __restrict__ bad, int max_tiles, int R, int r, int page_size, int num_pages,
                     int* err) {
  __shared__ long slot[BN];  // row of each key in the pools, -1: none
  __shared__ uint32_t half_bad[2];
  const int seq = singles + (int)blockIdx.y, ctx = ctx_len[seq], q_len = q_start[seq + 1] - q_start[seq];
  const int first = first_key(ctx, q_len, window), key0 = first + (int)blockIdx.x * BN;
  if (key0 >= ctx) return;
  const int row0 = first_row(q_start, ctx_len, singles, seq, window) + (int)blockIdx.x * BN;
  const int lo = window > 0 ? max(0, ctx - q_len - window + 1) : 0, n = min(BN, ctx - key0);
  const int tid = threadIdx.x;
  if (tid < BN) {
    const int key = key0 + tid;
    long at = -1;
    if (tid < n) {
      const int page = page_table[(size_t)seq * pt_stride + key / page_size];
      if (page >= 0 && page < num_pages)
        at = (long)page * page_size + key % page_size;
      else if (key >= lo)  // (in front of the window pages have been given back)
        atomicOr(err, DSP_ERR_BAD_PAGE);
    }
    slot[tid] = at;
    const uint32_t none = __ballot_sync(0xffffffffu, tid < n && at < 0);
    if ((tid & 31) == 0) half_bad[tid >> 5] = none;
  }
  __syncthreads();
  if (tid == 0)
    bad[(size_t)blockIdx.y * max_tiles + blockIdx.x] = (unsigned long long)half_bad[1] << 32 | half_bad[0];
  const int cp = R / 8, per = cp + r / 8;
  for (int i = tid; i < n * per; i += GATHER_THREADS) {
    const int j = i / per, c = i % per;
    const long at = slot[j];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (c < cp) {
      if (at >= 0) v = __ldg(reinterpret_cast<const uint4*>(c_pool + at * R) + c);
      reinterpret_cast<uint4*>(c_rows + (size_t)(row0 + j) * R)[c] = v;
    } else {
      if (at >= 0) v = __ldg(reinterpret_cast<const uint4*>(r_pool + at * r) + (c - cp));
      reinterpret_cast<uint4*>(r_rows + (size_t)(row0 + j) * r)[c - cp] = v;
    }
  }
}

// Latents [rows, R] and rotated parts [rows, 64] of the keys that the portions of prompts (sequences singles ..
// singles + portions - 1) see, one sequence after the other; bad [portions][max_tiles].
int gather(const void* c_pool, const void* r_pool, const int* page_table, int pt_stride, const int* q_start,
           const int* ctx_len, int singles, int portions, int window, void* c_rows, void* r_rows, void* bad, int max_tiles,
           int R, int page_size, int num_pages, int* err, cudaStream_t stream) {
  DSP_REQUIRE(R > 0 && R % 8 == 0 && max_tiles > 0 && portions <= 65535 && page_size > 0, "dsp_latent_prompts: R=%d, portions=%d", R, portions);
  DSP_REQUIRE(((uintptr_t)c_pool | (uintptr_t)r_pool | (uintptr_t)c_rows | (uintptr_t)r_rows) % 16 == 0,
              "dsp_latent_prompts: rows must be 16-byte aligned");
  DSP_CUDA(launch_plain(latent_gather_kernel, dim3(max_tiles, portions), dim3(GATHER_THREADS), 0, stream,
                        (const bf16*)c_pool, (const bf16*)r_pool, page_table, pt_stride, q_start, ctx_len, singles, window,
                        (bf16*)c_rows, (bf16*)r_rows, (unsigned long long*)bad, max_tiles, R, DR, page_size, num_pages, err));
  return 0;
}

// kv [rows, H * (DK + DV)]: every head's unrotated key, then every head's value, of the rows gathered above.
int attention(const Params& p, const void* kv, const void* r_rows, long rows, int num_tiles, int H, cudaStream_t stream) {
  DSP_REQUIRE(H > 0 && num_tiles <= 65535 && rows > 0 && p.scale_log2 > 0.f, "dsp_latent_prompts: %d heads, %d tiles", H, num_tiles);
  DSP_REQUIRE(p.rot >= 0 && p.rot <= DR && p.rot % 2 == 0 && (p.rot == 0 || p.inv_freq) && (p.layout == 0 || p.layout == 1) && p.window >= 0,
              "dsp_latent_prompts: rot=%d layout=%d window=%d", p.rot, p.layout, p.window);
  DSP_REQUIRE(p.q_stride % 8 == 0 && p.q_head_stride % 8 == 0 && p.qr_off % 8 == 0 && p.out_stride % 8 == 0 &&
                  ((uintptr_t)p.q | (uintptr_t)kv | (uintptr_t)r_rows | (uintptr_t)p.out) % 16 == 0,
              "dsp_latent_prompts: operands must be 16-byte aligned with strides in whole 16-byte pieces");
  const long columns = (long)H * (DK + DV);
  CUtensorMap map_k, map_r, map_v;
  DSP_REQUIRE(make_map_k_blocks(&map_k, kv, rows, columns, columns, BN, DK / 64) &&
                  make_map_k_blocks(&map_v, kv, rows, columns, columns, BN, DV / 64) &&
                  make_map(&map_r, r_rows, rows, DR, DR, BN),
              "dsp_latent_prompts: cannot encode the tensor maps");
  DSP_CUDA(cudaFuncSetAttribute(attn_latent_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  DSP_CUDA(launch_plain(attn_latent_prompt_kernel, dim3(H, num_tiles), dim3(THREADS), SMEM_BYTES, stream, p, map_k, map_r, map_v));
  return 0;
}
}  // namespace

extern "C" {
int dsp_gemm_stream(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                    long ldc, int M, int N, int K, int out_dtype, int target_ctas, int epilogue, long late_trigger_bytes,
                    const void* norm_src, long ld_src, float norm_eps, const void* gain2, void* C2, long ldc2,
                    cudaStream_t stream);
int dsp_gemm_tcgen05(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                     long ldc, int M, int N, int K, int out_dtype, int pair_mode, int epilogue, cudaStream_t stream);
int dsp_gemm_few_rows_faster(int M, int N, int K, int target_ctas);
}

// The three launches of a layer behind one call (called one by one from Python, with an allocation each, they cost
// the host some 30 us more than the three launches on the latents, and short portions are bound by the host): gathers the
// latents of the `rows` keys, expands them by `w_kv` [H * (DK + DV), R], on the product that ops/gemm.py would choose,
// and attends.  `work`: 2 room (R + 64 + H (DK + DV)) + 8 portions max_tiles bytes, room >= rows a multiple of 64.
extern "C" int dsp_latent_prompts(const void* c_pool, const void* r_pool, const int* page_table, int pt_stride,
                                  const int* q_start, const int* ctx_len, int singles, int portions, int window,
                                  const void* w_kv, void* work, long rows, long room, int max_tiles, int R, int page_size,
                                  int num_pages, const void* q, long q_stride, int q_head_stride, int qr_off,
                                  const float* inv_freq, int rot, int layout, float mag, const int* tile_seq,
                                  const int* tile_tok0, int num_tiles, void* out, long out_stride, const float* gate,
                                  long ldg, const float* sink, int H, float scale, int target_ctas, int always_few,
                                  long late_trigger_bytes, cudaStream_t stream) {
  if (portions <= 0 || num_tiles <= 0) return 0;
  DSP_REQUIRE(rows > 0 && rows <= room && room % 64 == 0 && room < (1l << 31), "dsp_latent_prompts: %ld rows in room for %ld", rows, room);
  int* err = dsp_device_error_ptr();
  DSP_REQUIRE(err != nullptr, "dsp_latent_prompts: no device error word");
  const int columns = H * (DK + DV);
  bf16* c_rows = (bf16*)work;
  bf16* r_rows = c_rows + room * R;
  bf16* kv = r_rows + room * DR;
  void* bad = kv + room * columns;
  int rc = gather(c_pool, r_pool, page_table, pt_stride, q_start, ctx_len, singles, portions, window, c_rows, r_rows, bad,
                  max_tiles, R, page_size, num_pages, err, stream);
  if (rc != 0) return rc;
  const int few = rows <= always_few ? 1 : dsp_gemm_few_rows_faster((int)rows, columns, R, target_ctas);
  if (few < 0) return few;
  rc = few ? dsp_gemm_stream(c_rows, R, w_kv, nullptr, nullptr, 0, kv, columns, (int)rows, columns, R, DSP_BF16, target_ctas, 0,
                             late_trigger_bytes, nullptr, 0, 0.f, nullptr, nullptr, 0, stream)
           : dsp_gemm_tcgen05(c_rows, R, w_kv, nullptr, nullptr, 0, kv, columns, (int)rows, columns, R, DSP_BF16, 1, 0, stream);
  if (rc != 0) return rc;
  Params p;
  p.q = (const bf16*)q;
  p.q_stride = q_stride;
  p.q_head_stride = q_head_stride;
  p.qr_off = qr_off;
  p.inv_freq = inv_freq;
  p.rot = rot;
  p.layout = layout;
  p.mag = mag;
  p.q_start = q_start;
  p.ctx_len = ctx_len;
  p.tile_seq = tile_seq;
  p.tile_tok0 = tile_tok0;
  p.tile_offset = singles;
  p.singles = singles;
  p.window = window;
  p.bad = (const unsigned long long*)bad;
  p.max_tiles = max_tiles;
  p.out = (bf16*)out;
  p.out_stride = out_stride;
  p.gate = gate;
  p.ldg = ldg;
  p.sink = sink;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.err = err;
  return attention(p, kv, r_rows, rows, num_tiles, H, stream);
}
