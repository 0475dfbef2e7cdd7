// C[M,N] = A[M,K] * W[N,K]^T (+ bias) (+ residual) for some hundred rows, bfloat16 in, 32-bit accumulation on the
// fifth-generation tensor cores: CTA pairs (cta_group::2) with the roles swapped.
//
// A tile is 256 rows of W (the lanes, 128 in each CTA of a pair) by a chunk of up to 256 rows of A (the columns, a
// multiple of 32): the rows of A are cut into equal chunks, so that 536 rows are computed as 3 x 192 and not as the
// 3 x 256 of gemm_tcgen05.cu, whose tiles have 256 rows of A.  Where there are few tiles, K is split over the pairs
// of a cluster (up to four) and every CTA adds and finishes its share of the tile's rows of A, read from the other
// pairs' shared memory in rank order.
//
// W and A come by TMA, two blocks of 64 k a request, into a ring of three slots; one thread of the pair issues the
// products into one of two accumulators in tensor memory; two groups of four warps take them 32 columns at a time through
// shared memory, so that a lane finishes four outputs of a row and a warp stores whole rows.  With programmatic dependent
// launch the first tiles of W are requested before the kernel waits for its predecessor.
//
// Every wait on an mbarrier is bounded; a wait that runs out is recorded in the device error word.
#include <atomic>

#include "tcgen05_common.cuh"

namespace {
using namespace tc;
constexpr int ROWS_W = 128, BK = 64, UMMA_K = 16, SUB = 2, SLOTS = 3, MAX_COLS = 256, MAX_SPLITS = 4;
constexpr int W_BYTES = ROWS_W * BK * 2;  // a CTA's rows of W, one block of k
constexpr int EPI_GROUPS = 2, EPI_WARPS = 4 * EPI_GROUPS, THREADS = 32 * (2 + EPI_WARPS);  // groups take chunks of columns in turn
constexpr int STAGING = EPI_GROUPS * 32 * ROWS_W * 4;  // a chunk of 32 columns as floats for each group
constexpr int TMEM_COLS = 512;                // two accumulators of up to 256 columns
constexpr int SMEM = SLOTS * SUB * (W_BYTES + MAX_COLS / 2 * BK * 2) + STAGING + 1024;
enum { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_GEGLU = 2, EPI_XIELU = 3 };

struct Args {
  int epilogue;
  const float* act;  // the two raw parameters of xIELU
  const bf16* bias;
  const void* residual;
  long ldr;
  void* C;
  long ldc;
  int M, N, K;
  int cols, chunk_rows, chunks;  // columns of a tile (rows of A, padded), rows of A it takes, tiles a block of W has
  int splits, slots_per_split;   // pairs that share a tile, ring slots (128 k) each of them takes
  int k_boxes;                   // one request brings both blocks of k of an operand
};

__device__ __forceinline__ void mbar_arrive_on(uint64_t* bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(mapa_u32(smem_u32(bar), rank)) : "memory");
}
__device__ __forceinline__ float4 load_remote(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                     __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(bf16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }

__device__ __forceinline__ float4 xielu4(float4 z, float ap, float an) {
  return make_float4(xielu_f(z.x, ap, an), xielu_f(z.y, ap, an), xielu_f(z.z, ap, an), xielu_f(z.w, ap, an));
}

// Four outputs of a row, this lane's n0 + 4 lane .. + 3, from their sums.
template <typename TOut>
__device__ __forceinline__ void finish_row(const Args& a, float4 v, int m, bool row_ok, int n4, float4 bias4, float4 res4) {
  if (!row_ok || n4 >= a.N) return;
  v.x = (v.x + bias4.x) + res4.x, v.y = (v.y + bias4.y) + res4.y;
  v.z = (v.z + bias4.z) + res4.z, v.w = (v.w + bias4.w) + res4.w;
  store4(reinterpret_cast<TOut*>(a.C) + (size_t)m * a.ldc + n4, v);
}
// Two rows of the gate/up product.  Of every 32 rows of W the first 16 are gates, the others the up rows of the same
// outputs: of eight lanes, 0..3 finish row m0 with what 4..7 hold of it, and these row m1 with what 0..3 hold.
template <typename TOut>
__device__ __forceinline__ void finish_units(const Args& a, float4 x0, float4 x1, int m0, int m1, bool ok0, bool ok1, int n0, int lane) {
  const bool low = (lane & 4) == 0, gelu = a.epilogue == EPI_GEGLU;
  const float4 mine = low ? x0 : x1, give = low ? x1 : x0;
  float4 got;
  got.x = __shfl_xor_sync(0xffffffffu, give.x, 4);
  got.y = __shfl_xor_sync(0xffffffffu, give.y, 4);
  got.z = __shfl_xor_sync(0xffffffffu, give.z, 4);
  got.w = __shfl_xor_sync(0xffffffffu, give.w, 4);
  const float4 gate = low ? mine : got, up = low ? got : mine;
  const int block = n0 + (lane >> 3) * 32;  // N is a multiple of 32: the block is whole or not there
  if ((low ? ok0 : ok1) && block < a.N)
    store4(reinterpret_cast<TOut*>(a.C) + (size_t)(low ? m0 : m1) * a.ldc + (block >> 1) + 4 * (lane & 3),
           make_float4(unit_times(gate.x, up.x, gelu), unit_times(gate.y, up.y, gelu), unit_times(gate.z, up.z, gelu),
                       unit_times(gate.w, up.w, gelu)));
}

template <typename TOut>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pairs_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const Args a, int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[SLOTS];   // used in the leader: both CTAs' loads land here
  __shared__ __align__(8) uint64_t empty_bar[SLOTS];  // one per CTA, freed by the multicast commit
  __shared__ __align__(8) uint64_t accum_full[2];     // one per CTA
  __shared__ __align__(8) uint64_t accum_empty[2];    // used in the leader: both CTAs' epilogue warps arrive
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank(), half = rank & 1, leader_rank = rank & ~1u;
  const int split = (int)(rank >> 1), group = 2 * a.splits;  // CTAs that share a tile
  const int first_tile = (int)blockIdx.x / group, stride = (int)gridDim.x / group;
  const int tiles = (a.N + 2 * ROWS_W - 1) / (2 * ROWS_W) * a.chunks;  // (block of W, chunk of rows), chunks innermost
  const int kb_begin = split * a.slots_per_split * SUB;
  const int num_kb = min((a.K + BK - 1) / BK - kb_begin, a.slots_per_split * SUB), num_steps = (num_kb + SUB - 1) / SUB;
  const int a_bytes = a.cols / 2 * BK * 2, slot_stride = SUB * (W_BYTES + a_bytes);  // a slot: blocks of W, then blocks of A

  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
    for (int b = 0; b < 2; ++b) mbar_init(&accum_full[b], 1), mbar_init(&accum_empty[b], 2 * EPI_WARPS);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    // W does not depend on the kernel before: its first tiles are asked for before the wait
    const bool leader = elect_one();
    const int ahead = first_tile < tiles ? min(num_steps, SLOTS) : 0;
    auto slot_bytes = [&](int st) { return 2 * (W_BYTES + a_bytes) * (a.k_boxes ? SUB : min(SUB, num_kb - st * SUB)); };
    auto load = [&](const CUtensorMap* map, unsigned char* dst, int bytes, uint64_t* bar, int st, int row0) {
      const int kb = kb_begin + st * SUB;
      if (a.k_boxes) {
        tma_load_3d_pair(dst, map, bar, 0, row0, kb);
      } else {
        for (int u = 0; u < SUB && st * SUB + u < num_kb; ++u) tma_load_2d_pair(dst + u * bytes, map, bar, (kb + u) * BK, row0);
      }
    };
    for (int st = 0; st < ahead; ++st) {
      const int w0 = (first_tile / a.chunks * 2 + (int)half) * ROWS_W;
      if (leader) {
        if (half == 0) mbar_expect_tx(&full_bar[st], slot_bytes(st));
        load(&map_w, smem + st * slot_stride, W_BYTES, &full_bar[st], st, w0);
      }
    }
    pdl_wait();
    int it = 0, s = 0, phase = 1;
    for (int tile = first_tile; tile < tiles && !failed; tile += stride) {
      const int w0 = (tile / a.chunks * 2 + (int)half) * ROWS_W, m0 = tile % a.chunks * a.chunk_rows + (int)half * (a.cols / 2);
      for (int st = 0; st < num_steps; ++st, ++it) {
        unsigned char* slot = smem + s * slot_stride;
        if (it >= ahead) {
          if (!mbar_wait(&empty_bar[s], phase)) {
            failed = 1;
            break;
          }
          if (leader) {
            if (half == 0) mbar_expect_tx(&full_bar[s], slot_bytes(st));
            load(&map_w, slot, W_BYTES, &full_bar[s], st, w0);
          }
        }
        if (leader) load(&map_a, slot + SUB * W_BYTES, a_bytes, &full_bar[s], st, m0);
        if (++s == SLOTS) s = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    if (half == 0) {
      const bool leader = elect_one();
      const uint32_t idesc = umma_idesc(2 * ROWS_W, a.cols);  // M 256 across the pair
      const uint16_t mask = (uint16_t)(3u << leader_rank);
      int s = 0, phase = 0, local = 0;
      for (int tile = first_tile; tile < tiles && !failed; tile += stride, ++local) {
        const int buf = local & 1;
        bool ok = mbar_wait(&accum_empty[buf], ((local >> 1) & 1) ^ 1);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * MAX_COLS);
        for (int st = 0; st < num_steps && ok; ++st) {
          ok = mbar_wait(&full_bar[s], phase);
          if (!ok) break;
          tc_fence_after();
          const int subs = min(SUB, num_kb - st * SUB);
          const uint64_t w = umma_desc(smem_u32(smem + s * slot_stride)), x = w + (SUB * W_BYTES >> 4);
          if (leader) {
#pragma unroll
            for (int u = 0; u < SUB; ++u) {
              if (u >= subs) break;
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k)
                umma_pair(tmem_d, w + (u * (W_BYTES >> 4) + k * 2), x + (u * (a_bytes >> 4) + k * 2), idesc, (st | u | k) != 0);
            }
            umma_commit_pair(&empty_bar[s], mask);
          }
          if (++s == SLOTS) s = 0, phase ^= 1;
        }
        if (!ok) {
          failed = 1;
          break;
        }
        if (leader) umma_commit_pair(&accum_full[buf], mask);
      }
    }
  } else {
    pdl_wait();  // the residual comes from earlier kernels, and C may still be read by them
    const int quarter = warp & 3, ew = (warp - 2) & 3, eg = (warp - 2) >> 2;
    float* staging = reinterpret_cast<float*>(smem + SLOTS * slot_stride) + eg * 32 * ROWS_W;
    int local = 0;
    for (int tile = first_tile; tile < tiles; tile += stride, ++local) {
      const int buf = local & 1;
      const int n0 = (tile / a.chunks * 2 + (int)half) * ROWS_W, m0 = tile % a.chunks * a.chunk_rows;
      const int rows = min(a.chunk_rows, a.M - m0), n4 = n0 + 4 * lane;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * MAX_COLS);
      if (a.splits > 1) {
        if (!__all_sync(0xffffffffu, mbar_wait(&accum_full[buf], (local >> 1) & 1))) {
          failed = 1;
          break;
        }
        tc_fence_after();
        // this pair's sums into the drained ring, [row of A][128]
        float* part = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
#pragma unroll 1
        for (int c0 = 32 * eg; c0 < rows; c0 += 32 * EPI_GROUPS) {
          uint32_t v[32];
          tmem_ld32(taddr + (uint32_t)c0, v);
#pragma unroll
          for (int c = 0; c < 32; ++c) part[(c0 + c) * ROWS_W] = __uint_as_float(v[c]);
        }
        continue;
      }
      float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f), res4[8];
      if (a.bias && n4 < a.N) bias4 = load4(a.bias + n4);
      const float ap = a.act ? softplus_f(a.act[0]) : 0.f, an = a.act ? 0.5f + softplus_f(a.act[1]) : 0.f;
      auto fetch_residual = [&](int c0) {  // of the rows this warp finishes in the chunk at c0
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int m = c0 + 8 * ew + i;
          res4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (a.residual && m < rows && n4 < a.N) res4[i] = load4(reinterpret_cast<const TOut*>(a.residual) + (size_t)(m0 + m) * a.ldr + n4);
        }
      };
      fetch_residual(32 * eg);
      if (!__all_sync(0xffffffffu, mbar_wait(&accum_full[buf], (local >> 1) & 1))) {
        failed = 1;
        break;
      }
      tc_fence_after();
      uint32_t v[32];
      if (32 * eg < rows) tmem_ld32_nowait(taddr + (uint32_t)(32 * eg), v);
#pragma unroll 1
      for (int c0 = 32 * eg; c0 < rows; c0 += 32 * EPI_GROUPS) {
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) staging[c * ROWS_W + quarter * 32 + lane] = __uint_as_float(v[c]);
        if (c0 + 32 * EPI_GROUPS < rows) tmem_ld32_nowait(taddr + (uint32_t)(c0 + 32 * EPI_GROUPS), v);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + eg) : "memory");
        float4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(staging + (8 * ew + i) * ROWS_W + 4 * lane);
        if (a.epilogue == EPI_XIELU) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int m = c0 + 8 * ew + i;
            const float4 y = xielu4(x[i], ap, an);
            if (m < rows && n4 < a.N) store4(reinterpret_cast<TOut*>(a.C) + (size_t)(m0 + m) * a.ldc + n4, y);
          }
        } else if (a.epilogue != EPI_PLAIN) {
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const int m = c0 + 8 * ew + i;
            finish_units<TOut>(a, x[i], x[i + 1], m0 + m, m0 + m + 1, m < rows, m + 1 < rows, n0, lane);
          }
        } else {
          float4 now[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) now[i] = res4[i];
          if (c0 + 32 * EPI_GROUPS < rows) fetch_residual(c0 + 32 * EPI_GROUPS);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int m = c0 + 8 * ew + i;
            finish_row<TOut>(a, x[i], m0 + m, m < rows, n4, bias4, now[i]);
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + eg) : "memory");  // the staged chunk has been read
      }
      // the accumulator has been read
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_on(&accum_empty[buf], leader_rank);
    }
  }

  if (a.splits > 1) {
    // one tile a cluster: its CTAs that hold the same rows of W finish the rows of A in turn
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    pdl_wait();
    if (!failed) {
      const int n0 = (first_tile / a.chunks * 2 + (int)half) * ROWS_W, m0 = first_tile % a.chunks * a.chunk_rows;
      const int rows = min(a.chunk_rows, a.M - m0), n4 = n0 + 4 * lane;
      float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.bias && n4 < a.N) bias4 = load4(a.bias + n4);
      const float ap = a.act ? softplus_f(a.act[0]) : 0.f, an = a.act ? 0.5f + softplus_f(a.act[1]) : 0.f;
      uint32_t from[MAX_SPLITS];
#pragma unroll
      for (int sp = 0; sp < MAX_SPLITS; ++sp) from[sp] = sp < a.splits ? mapa_u32(smem_u32(smem) + lane * 16, 2 * sp + half) : 0;
      auto total_of = [&](int m) {
        float4 part[MAX_SPLITS];
#pragma unroll
        for (int sp = 0; sp < MAX_SPLITS; ++sp)
          if (sp < a.splits) part[sp] = load_remote(from[sp] + m * (ROWS_W * 4));
        float4 total = part[0];
#pragma unroll
        for (int sp = 1; sp < MAX_SPLITS; ++sp)
          if (sp < a.splits) total.x += part[sp].x, total.y += part[sp].y, total.z += part[sp].z, total.w += part[sp].w;
        return total;
      };
      // rows split, split + splits, ...: a warp takes four at a time, their loads side by side
      for (int r0 = 4 * warp; split + a.splits * r0 < rows; r0 += 4 * (THREADS / 32)) {
        float4 x[4], res4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = min(split + a.splits * (r0 + i), rows - 1);
          res4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (a.residual && n4 < a.N) res4[i] = load4(reinterpret_cast<const TOut*>(a.residual) + (size_t)(m0 + m) * a.ldr + n4);
          x[i] = total_of(m);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = split + a.splits * (r0 + i);
          if (a.epilogue == EPI_XIELU) x[i] = xielu4(x[i], ap, an);
          if (a.epilogue == EPI_PLAIN || a.epilogue == EPI_XIELU) finish_row<TOut>(a, x[i], m0 + m, m < rows, n4, bias4, res4[i]);
        }
        if (a.epilogue == EPI_SWIGLU || a.epilogue == EPI_GEGLU) {
#pragma unroll
          for (int i = 0; i < 4; i += 2) {
            const int m = split + a.splits * (r0 + i);
            finish_units<TOut>(a, x[i], x[i + 1], m0 + m, m0 + m + a.splits, m < rows, m + a.splits < rows, n0, lane);
          }
        }
      }
    }
  }
  __syncthreads();
  if (failed) {
    if (threadIdx.x == 0) atomicOr(err, DSP_ERR_WAIT_LIMIT);
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
  tc_fence_before();
  cluster_sync_all();  // the peers are done with this CTA's shared memory and barriers
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

template <typename TOut>
cudaError_t launch(int clusters, int splits, const CUtensorMap& map_a, const CUtensorMap& map_w, const Args& a, int* err,
                   cudaStream_t stream, int* fit) {
  auto kernel = gemm_pairs_kernel<TOut>;
  static std::atomic<bool> configured[MAX_DEVICES] = {};
  const int device = current_device();
  if (device < 0) return cudaErrorInvalidDevice;
  if (!configured[device].load(std::memory_order_relaxed)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured[device].store(true, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * 2 * splits, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = fit ? 1 : 2;
  if (fit) return cudaOccupancyMaxActiveClusters(fit, kernel, &cfg);
  return cudaLaunchKernelEx(&cfg, kernel, map_a, map_w, a, err);
}

// fits[s]: clusters of s pairs that the device holds at once (a cluster stays inside a group of SMs, so fewer large ones fit
// than there are SMs; 0: none does).  Asked once a device; an answer that does not come is an error of this call (false,
// with the message set) and nothing that is remembered.
struct Fits {
  int of[MAX_SPLITS + 1];
};
bool clusters_that_fit(Fits& fits) {
  static std::atomic<int> known[MAX_DEVICES][MAX_SPLITS + 1] = {};  // one more than the answer, 0: not asked
  const int device = current_device();
  for (int splits = 1; splits <= MAX_SPLITS; ++splits) {
    int n = device < 0 ? 0 : known[device][splits].load(std::memory_order_relaxed) - 1;
    if (device < 0 || n < 0) {
      n = 0;
      const CUtensorMap none = {};
      const cudaError_t e = launch<bf16>(1, splits, none, none, Args{}, nullptr, nullptr, &n);
      if (e != cudaSuccess) {
        dsp_set_error("dsp_gemm_pairs: how many clusters of %d pairs fit is not known (%s)", splits, cudaGetErrorString(e));
        cudaGetLastError();
        return false;
      }
      known[device][splits].store(n + 1, std::memory_order_relaxed);
    }
    fits.of[splits] = n;
  }
  return true;
}

struct Plan {
  int cols, chunk_rows, chunks, splits, slots_per_split, clusters;
  double us;  // estimate; negative: none (the message is set where `splits` is 0)
};
Plan make_plan(int M, int N, int K, const Fits& fits, int force_splits, int force_chunks);
// The plan of a size, of which the thread's last few are remembered: the layers of a step ask for the same ones.
Plan plan_of(int M, int N, int K, int splits, int chunks) {
  struct Known {
    int M, N, K, device;
    Plan plan;
  };
  constexpr int KEPT = 32;
  static thread_local Known known[KEPT] = {};
  static thread_local int next = 0;
  const int device = current_device();
  const bool chosen = splits == 0 && chunks == 0 && device >= 0;
  if (chosen)
    for (const Known& k : known)
      if (k.M == M && k.N == N && k.K == K && k.device == device) return k.plan;
  Fits fits;
  if (!clusters_that_fit(fits)) return Plan{0, 0, 0, 0, 0, 0, -1.0};
  const Plan p = make_plan(M, N, K, fits, splits, chunks);
  if (chosen && p.us >= 0.0) known[next++ % KEPT] = {M, N, K, device, p};
  return p;
}
// Chunks of rows and splits of K by an estimate in microseconds, fitted on launches that follow one another in a graph
// and read W from memory: 15 shapes from 2,304 x 768 to 37,888 x 3,584, 72 to 2,048 rows, every split and number of chunks
// (rms error 5 %).  A ring slot costs more the more columns and the more pairs are busy, a tile its epilogue.
Plan make_plan(int M, int N, int K, const Fits& fits, int force_splits, int force_chunks) {
  Plan best = {};
  best.us = -1.0, best.splits = 1;
  const int blocks = (N + 2 * ROWS_W - 1) / (2 * ROWS_W), slots = (K + SUB * BK - 1) / (SUB * BK);
  const int least = (M + MAX_COLS - 1) / MAX_COLS, pairs = fits.of[1];
  const double w_us = 2.0 * N * K / 6.5e6;  // W at the memory's rate
  for (int splits = 1; splits <= MAX_SPLITS; ++splits) {
    const int fit = fits.of[splits];
    if (fit <= 0 || (force_splits > 0 && splits != force_splits)) continue;
    if (splits > 1 && slots < 2 * splits) break;
    for (int chunks = least; chunks < least + 3; ++chunks) {
      if (force_chunks > 0 && chunks != force_chunks) continue;
      Plan p;
      p.chunk_rows = (M + chunks - 1) / chunks;
      p.cols = (p.chunk_rows + 31) / 32 * 32;
      p.chunks = (M + p.chunk_rows - 1) / p.chunk_rows;
      p.slots_per_split = (slots + splits - 1) / splits;
      p.splits = (slots + p.slots_per_split - 1) / p.slots_per_split;
      if (p.splits != splits) continue;
      const long tiles = (long)blocks * p.chunks;
      if (splits > 1 && tiles > fit) continue;
      p.clusters = (int)(tiles < fit ? tiles : fit);
      const double rounds = (double)((tiles + fit - 1) / fit), c = p.cols / 256.0;
      const double busy = tiles * splits < pairs ? (double)tiles * splits / pairs : 1.0;
      p.us = 2.22 + rounds * (p.slots_per_split * (0.315 - 0.022 * busy + c * (0.183 + 0.138 * busy)) - 0.55) + 8.94 * c +
             (splits > 1 ? 1.85 - 3.37 * c : 0.0) + 0.5 * w_us;
      if (best.us < 0.0 || p.us < best.us) best = p;
    }
  }
  return best;
}
}  // namespace

extern "C" int dsp_gemm_other_rows(int M, int N, int K, int target_ctas, int result, double* us, int* k_blocks_in_a_row);

// The time of this product for a bfloat16 result (0), one of 32 bits (1), a gated one (2) or one that xIELU is applied to (3),
// fitted as dsp_gemm_other_rows is; rms error 7 %.
static double time_us(const Plan& p, int N, int K, int target_ctas, int result) {
  static constexpr double FIT[4][11] = {{4.592, -1.518, 0.131, 0.208, 0.319, -0.049, 4.186, 0.642, -1.413, 0.411, 3.534},
                                        {5.056, -1.721, 0.144, 0.188, 0.282, 0.016, 3.055, 0.356, -0.941, 0.418, 4.389},
                                        {4.822, -1.399, 0.123, 0.212, 0.345, -0.063, 3.618, 0.362, 0.201, 0.391, 2.827},
                                        {6.424, -3.517, 0.069, 0.352, 0.613, -0.469, 3.181, 1.244, -7.046, 0.365, 13.721}};
  const long tiles = (long)((N + 2 * ROWS_W - 1) / (2 * ROWS_W)) * p.chunks;
  const double rounds = (double)((tiles + p.clusters - 1) / p.clusters), slots = p.slots_per_split, cols = p.cols / 256.0;
  const double busy = fmin(1.0, 2.0 * tiles * p.splits / target_ctas), split = p.splits > 1;
  const double* c = FIT[result];
  return c[0] + rounds * (c[1] + slots * (c[2] + c[3] * busy + cols * (c[4] + c[5] * busy)) + c[10] * cols) + c[6] * cols +
         split * (c[7] + c[8] * cols) + c[9] * 2.0 * N * K / 6.5e6;
}
// Whether this product beats what runs otherwise (-1: not known, the message is set): the few-row or the many-row kernel for
// results 0 to 2, with a margin for the fits' errors (of 3,432 sizes eight take more than 1.03 of the other kernel's time, at
// most 1.11; the mean is 0.961 / 0.927 / 0.897 of it), and for 3 a product with a 32-bit result and the activation behind it (mean
// 0.88, at most 1.15).  32-bit results stay where their sums are shorter: the tensor cores cut every one off (300 rows x 2,048
// x 8,960: 3.2e-6 off 64 bits here, 2.3e-6 in the few-row kernel, which splits K further, 1.0e-5 in the many-row one).  This,
// few-row and many-row: 536 rows x 1,536 x 1,536 9.8 / 11.8 / 11.8 us, x 17,920 x 1,536 29.0 / 30.7 / 30.5, x 1,536 x 8,960 21.3 /
// 23.1 / 42.3; 1,016 rows x 3,584 x 18,944 104.5 / 169 / 108, x 2,048 x 1,536 13.6 / 13.2 / 11.3.
extern "C" int dsp_gemm_pairs_faster(int M, int N, int K, int target_ctas, int result) {
  if (M <= 0 || M > 2048 || N <= 0 || K <= 0 || target_ctas <= 0 || result < 0 || result > 3) return 0;  // (fitted up to there)
  double other = 0.0;
  int in_a_row = 0;
  const int rc = dsp_gemm_other_rows(M, N, K, target_ctas, result == 3 ? 1 : result, &other, &in_a_row);
  if (rc != 0) return rc;
  const Plan p = plan_of(M, N, K, 0, 0);
  if (p.splits == 0) return -1;
  if (p.us < 0.0) return 0;
  const double us = time_us(p, N, K, target_ctas, result);
  if (result == 0) return us < 0.955 * other;
  if (result == 2) return us < 0.94 * other;
  const bool no_longer_sums = p.slots_per_split * SUB <= in_a_row;
  if (result == 1) return no_longer_sums && us < 0.94 * other;
  const double here = time_us(p, N, K, target_ctas, 1);  // of the 32-bit product that the activation would follow
  const double product = no_longer_sums && here < 0.94 * other ? here : other;
  return us < 3.22 + 1.063 * product + 1.493e-6 * M * N;
}

// The plan of a size where fits[0..3] clusters of one to four pairs fit: pairs that share a tile, chunks of rows, clusters
// launched (1: there is none).
extern "C" int dsp_gemm_pairs_plan(int M, int N, int K, const int* fits, int* plan) {
  Fits f = {};
  for (int s = 1; s <= MAX_SPLITS; ++s) f.of[s] = fits[s - 1];
  const Plan p = make_plan(M, N, K, f, 0, 0);
  if (p.us < 0.0) return 1;
  plan[0] = p.splits, plan[1] = p.chunks, plan[2] = p.clusters;
  return 0;
}

// Operands as dsp_gemm_tcgen05 takes them; N, ldc and ldr multiples of 4, C and residual on 16 bytes (bfloat16: 8),
// bias on 8.  epilogue 3: xIELU of every output, its two raw parameters in `act` (null otherwise).  splits, chunks: pairs that share a tile's K, chunks of rows (0: by the estimate).
extern "C" int dsp_gemm_pairs(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                              long ldc, int M, int N, int K, int out_dtype, int epilogue, const float* act,
                              int splits, int chunks, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  DSP_REQUIRE(K > 0 && K % 8 == 0 && lda % 8 == 0, "dsp_gemm_pairs: K=%d and the row stride must be multiples of 8", K);
  DSP_REQUIRE(((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0, "dsp_gemm_pairs: operands must be 16-byte aligned");
  DSP_REQUIRE(out_dtype == DSP_BF16 || out_dtype == DSP_F32, "dsp_gemm_pairs: unknown output dtype %d", out_dtype);
  DSP_REQUIRE(epilogue >= EPI_PLAIN && epilogue <= EPI_XIELU, "dsp_gemm_pairs: unknown epilogue %d", epilogue);
  DSP_REQUIRE(epilogue == EPI_PLAIN || ((epilogue == EPI_XIELU || N % 32 == 0) && bias == nullptr && residual == nullptr),
              "dsp_gemm_pairs: an activation takes no bias or residual, and a gated one N in whole blocks of 32");
  DSP_REQUIRE((epilogue == EPI_XIELU) == (act != nullptr), "dsp_gemm_pairs: xIELU and its parameters come together");
  const uintptr_t mask = out_dtype == DSP_F32 ? 15 : 7;
  DSP_REQUIRE(N % 4 == 0 && ldc % 4 == 0 && ((uintptr_t)C & mask) == 0 && (residual == nullptr || (ldr % 4 == 0 && ((uintptr_t)residual & mask) == 0)) &&
                  (bias == nullptr || ((uintptr_t)bias & 7) == 0),
              "dsp_gemm_pairs: rows of four outputs (N=%d, ldc=%ld)", N, ldc);
  int* err = dsp_device_error_ptr();
  DSP_REQUIRE(err != nullptr, "dsp_gemm_pairs: no device error word");
  const Plan p = plan_of(M, N, K, splits, chunks);
  if (p.splits == 0) return -1;
  DSP_REQUIRE(p.us >= 0.0, "dsp_gemm_pairs: no plan for M=%d, N=%d, K=%d in %d splits and %d chunks", M, N, K, splits, chunks);
  Args a = {epilogue, act, (const bf16*)bias, residual, ldr, C, ldc, M, N, K, p.cols, p.chunk_rows, p.chunks, p.splits, p.slots_per_split, 0};
  CUtensorMap map_a, map_w;
  a.k_boxes = make_map_k_blocks(&map_a, A, M, K, lda, p.cols / 2, SUB) && make_map_k_blocks(&map_w, W, N, K, K, ROWS_W, SUB);
  if (!a.k_boxes) {
    DSP_REQUIRE(make_map(&map_a, A, M, K, lda, p.cols / 2), "dsp_gemm_pairs: cannot encode the tensor map of A");
    DSP_REQUIRE(make_map(&map_w, W, N, K, K, ROWS_W), "dsp_gemm_pairs: cannot encode the tensor map of W");
  }
  DSP_CUDA(out_dtype == DSP_BF16 ? launch<bf16>(p.clusters, p.splits, map_a, map_w, a, err, stream, nullptr)
                                 : launch<float>(p.clusters, p.splits, map_a, map_w, a, err, stream, nullptr));
  return 0;
}
