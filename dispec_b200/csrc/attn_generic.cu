// Causal grouped-query attention over the paged key/value cache, all arithmetic in 32-bit.
//
// The G = H / KVH query heads of a group, and in heads of up to 128 dimensions several tokens of a portion as
// well, share every key and value load (the two kernels: below).  The query at absolute position p sees keys b with
//     max(0, p - window + 1) <= b <= p        (window == 0: every key from 0)
// which is the lower-right aligned causal mask for a portion of a prompt on top of cached
// tokens, and a single decoded token alike.  Online softmax (running max m, running sum l)
// over tiles of 128 or 64 keys.  Keys have D dimensions and values Dv (the pools have their own widths).
// With `mask_mode` 1 the number `window` is a chunk size instead: position p sees the keys of its own
// chunk, floor(p / size) * size <= b <= p (chunks counted from position 0 of the sequence).
// With `keep_first` = F the keys b < F are seen as well, however far behind the window they lie.
// With `sink` the softmax has one more, imaginary key and no value for it: the weights are
// exp(s_j) / (exp(z) + sum exp(s_j)), z = sink_values[head] (unscaled), or 0 without `sink_values`;
// the running pair starts at (m, l) = (z, 1) instead of (-inf, 0).
// With `turn_freq` (float [Dv/2]) the result of every head is turned back: pair (m, m + Dv/2) by
// -p * turn_freq[m] (the values were stored turned by their own positions).  With `gate` (float, row stride ldg, laid
// out like the output's columns) every result is multiplied by the sigmoid of its gate value.  Any head_dim that is a multiple of 4 (float) / 8 (bfloat16) up to
// 512, any G.  This kernel is the attention of the 32-bit path and the fallback of the
// bfloat16 path for head sizes the tensor-core kernel is not built for.
//
// q:   element (t, head, d) at q[t * q_stride + head * D + d]
// out: element (t, head, d) at out[t * out_stride + head * Dv + d]
// pools: [num_pages, KVH, page_size, D] (keys) and [..., Dv] (values); page = page_table[seq * pt_stride + b / page_size]
//
// Two kernels.  `attn_rows_kernel` takes heads of up to 128 dimensions in rows of whole 16-byte (bfloat16: 8-byte)
// pieces: several tokens of a portion share every key and value, which pass through shared memory.
// `attn_generic_kernel` takes the rest, one block per (query token, KV head).
#include <type_traits>

#include "common.cuh"

namespace {
constexpr int THREADS = 128;   // = keys per tile
constexpr int GCHUNK = 8;      // query heads handled per pass
constexpr int DPT = 4;         // output dims per thread: head_dim <= THREADS * DPT

template <typename T>
__global__ void __launch_bounds__(THREADS)
attn_generic_kernel(const T* __restrict__ q, long q_stride, const T* __restrict__ k_pool,
                    const T* __restrict__ v_pool, const int* __restrict__ page_table,
                    int pt_stride, const int* __restrict__ positions,
                    const int* __restrict__ seq_of_token, void* __restrict__ out, int out_dtype, long out_stride,
                    int H, int KVH, int D, int Dv, int page_size, int num_pages, int window, int mask_mode,
                    int keep_first, float scale, int sink, const float* __restrict__ sink_values,
                    const float* __restrict__ turn_freq, const float* __restrict__ gate, long ldg, int* err) {
  extern __shared__ float smem[];
  float* qs = smem;                       // [GCHUNK][D]
  float* ps = qs + GCHUNK * D;            // [GCHUNK][THREADS]
  long* slot = (long*)(ps + GCHUNK * THREADS);  // [THREADS] row of each key in the pools (-1: none)
  float* os = (float*)(slot + THREADS);   // [GCHUNK][Dv] results before they are turned back (with turn_freq)
  __shared__ float red[GCHUNK][THREADS / 32];

  const int t = blockIdx.x, kvh = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pos = positions[t];
  if (pos < 0) return;
  const int seq = seq_of_token[t];
  const int G = H / KVH;
  int lo = window > 0 ? (mask_mode == 1 ? (pos / window) * window : max(0, pos - window + 1)) : 0;
  if (lo <= keep_first) lo = 0;
  const int front = min(keep_first, lo), nfront = (front + THREADS - 1) / THREADS;  // kept keys, and the tiles they take
  const int hi = pos, ntiles = nfront + (hi - lo) / THREADS + 1;
  const int* table = page_table + (size_t)seq * pt_stride;

  for (int g0 = 0; g0 < G; g0 += GCHUNK) {
    const int gn = min(GCHUNK, G - g0);
    __syncthreads();
    for (int i = tid; i < gn * D; i += THREADS) {
      const int g = i / D, d = i % D;
      qs[g * D + d] = to_f32(q[(size_t)t * q_stride + (size_t)(kvh * G + g0 + g) * D + d]) * scale;
    }
    float m[GCHUNK], l[GCHUNK], acc[GCHUNK][DPT];
#pragma unroll
    for (int g = 0; g < GCHUNK; ++g) {
      m[g] = sink ? ((sink_values && g < gn) ? sink_values[kvh * G + g0 + g] : 0.f) : -INFINITY;
      l[g] = sink ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < DPT; ++j) acc[g][j] = 0.f;
    }
    __syncthreads();

    for (int tile = 0; tile < ntiles; ++tile) {
      const int kt = tile < nfront ? tile * THREADS : lo + (tile - nfront) * THREADS;
      const int last = tile < nfront ? front - 1 : hi;
      const int key = kt + tid;
      const bool valid = key <= last;
      float s[GCHUNK];
#pragma unroll
      for (int g = 0; g < GCHUNK; ++g) s[g] = -INFINITY;
      long off = -1;
      if (valid) {
        const int page = table[key / page_size];
        if (page < 0 || page >= num_pages) {
          atomicOr(err, DSP_ERR_BAD_PAGE);
        } else {
          off = ((long)page * KVH + kvh) * page_size + (key % page_size);
          const T* kr = k_pool + off * D;
#pragma unroll
          for (int g = 0; g < GCHUNK; ++g) s[g] = 0.f;
          for (int d = 0; d < D; ++d) {
            const float kv = to_f32(kr[d]);
#pragma unroll
            for (int g = 0; g < GCHUNK; ++g)
              if (g < gn) s[g] = fmaf(qs[g * D + d], kv, s[g]);
          }
        }
      }
      slot[tid] = off;
      // tile maxima, one per head
#pragma unroll
      for (int g = 0; g < GCHUNK; ++g) {
        const float wm = warp_max(s[g]);
        if (lane == 0) red[g][warp] = wm;
      }
      __syncthreads();
      float alpha[GCHUNK], p[GCHUNK];
#pragma unroll
      for (int g = 0; g < GCHUNK; ++g) {
        float tm = red[g][0];
#pragma unroll
        for (int w = 1; w < THREADS / 32; ++w) tm = fmaxf(tm, red[g][w]);
        const float m_new = fmaxf(m[g], tm);
        // m_new stays -inf only for heads beyond gn or when every page id was bad
        alpha[g] = (m_new == -INFINITY) ? 1.f : expf(m[g] - m_new);
        p[g] = (off >= 0 && g < gn) ? expf(s[g] - m_new) : 0.f;
        m[g] = m_new;
        ps[g * THREADS + tid] = p[g];
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GCHUNK; ++g) {
        const float ws = warp_sum(p[g]);
        if (lane == 0) red[g][warp] = ws;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GCHUNK; ++g) {
        float ts = red[g][0];
#pragma unroll
        for (int w = 1; w < THREADS / 32; ++w) ts += red[g][w];
        l[g] = l[g] * alpha[g] + ts;
#pragma unroll
        for (int j = 0; j < DPT; ++j) acc[g][j] *= alpha[g];
      }
      // weighted sum of values: thread owns dims tid, tid+128, ...
      const int nkeys = min(THREADS, last - kt + 1);
      for (int j = 0; j < nkeys; ++j) {
        const long vo = slot[j];
        if (vo < 0) continue;
        const T* vr = v_pool + vo * Dv;
#pragma unroll
        for (int dd = 0; dd < DPT; ++dd) {
          const int d = tid + dd * THREADS;
          if (d < Dv) {
            const float vv = to_f32(vr[d]);
#pragma unroll
            for (int g = 0; g < GCHUNK; ++g)
              if (g < gn) acc[g][dd] = fmaf(ps[g * THREADS + j], vv, acc[g][dd]);
          }
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int g = 0; g < GCHUNK; ++g) {
      if (g >= gn) continue;
      const float inv = l[g] > 0.f ? 1.f / l[g] : 0.f;
#pragma unroll
      for (int dd = 0; dd < DPT; ++dd) {
        const int d = tid + dd * THREADS;
        if (d >= Dv) continue;
        const size_t col = (size_t)(kvh * G + g0 + g) * Dv + d;
        float y = acc[g][dd] * inv;
        if (gate) y /= 1.f + expf(-gate[(size_t)t * ldg + col]);
        if (turn_freq)
          os[g * Dv + d] = y;
        else
          st_any(out, out_dtype, (size_t)t * out_stride + col, y);
      }
    }
    if (turn_freq) {
      __syncthreads();
      const int half = Dv / 2;
      for (int i = tid; i < gn * Dv; i += THREADS) {
        const int g = i / Dv, d = i % Dv;
        const int mth = d < half ? d : d - half;
        float sn, cn;
        sincosf((float)pos * turn_freq[mth], &sn, &cn);
        // the inverse turn: (u, v) -> (u cos + v sin, v cos - u sin)
        const float v = d < half ? os[i] * cn + os[i + half] * sn : os[i] * cn - os[i - half] * sn;
        st_any(out, out_dtype, (size_t)t * out_stride + (size_t)(kvh * G + g0 + g) * Dv + d, v);
      }
    }
  }
}

// ------------------------------------------------------------------ heads of up to 128 dimensions
// One block per (run of query tokens, KV head).  A run: tokens of one sequence at neighbouring positions, cut
// where a position is a multiple of the `per` tokens whose G query heads fill the block's rows; the grid has a
// block per token, and those whose token does not begin a run leave at once.  Row r of the block is head
// g0 + r % gn of token r / gn.  A thread owns RI rows x KJ keys of the scores and RI rows x 4 DJ dimensions of
// the result (the same rows, so the running maximum and sum stay in its registers); the keys of the next tile
// are on their way while the values of this one are summed, and the other way round.
//
// What bounds it: the latencies of a tile, one after the other (a block alone on an SM takes 7 us a tile of 16 rows, 11 of
// 32, the FMA units 1 and 2).  260 tokens of a prompt beside four single tokens at 330, 12 heads of 128 on 2 KV heads:
// 55 us; 75 with 128 threads and runs of 32 rows (`rows_kernel` has the other sizes), 299 with a block per token whose
// threads each walk a key of their own through global memory.
constexpr int TILE_KEYS = 64, MAX_DIM = 128;

struct RowsArgs {
  const void *q, *k_pool, *v_pool;
  const int *page_table, *positions, *seq_of_token;
  void* out;
  const float *sink_values, *turn_freq, *gate;
  long q_stride, out_stride, ldg;
  int pt_stride, T, H, KVH, D, Dv, page_size, num_pages, window, mask_mode, keep_first, sink, out_dtype;
  float scale;
  int* err;
};

// Four neighbouring elements as floats in shared memory: an asynchronous copy, or a load and a conversion.
__device__ __forceinline__ void bring4(float* dst, const float* src, bool there) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void bring4(float* dst, const bf16* src, bool there) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (there) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(src);
    const float2 a = __bfloat1622float2(p[0]), b = __bfloat1622float2(p[1]);
    v = make_float4(a.x, a.y, b.x, b.y);
  }
  *reinterpret_cast<float4*>(dst) = v;
}
__device__ __forceinline__ void end_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_groups() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// R rows on a grid of TY x TX of NT threads.
template <typename T, int R, int TY, int NT>
__device__ __forceinline__ void attn_rows(const RowsArgs& a, float* smem, int t0, int n, int pos0, int seq, int kvh,
                                          int g0, int gn) {
  constexpr int TX = NT / TY, RI = R / TY, KJ = TILE_KEYS / TX, DJ = MAX_DIM / (4 * TX), LP = TILE_KEYS + 4;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int D = a.D, Dv = a.Dv, LK = D + 4, LV = Dv + 4, G = a.H / a.KVH, rows = n * gn;
  float* qs = smem;                     // [R][LK]
  float* ks = qs + R * LK;              // [TILE_KEYS][LK]
  float* vs = ks + TILE_KEYS * LK;      // [TILE_KEYS][LV]
  float* ps = vs + TILE_KEYS * LV;      // [R][LP]
  long* slot = (long*)(ps + R * LP);    // [2][TILE_KEYS] row of each key of a tile in the pools, -1: none
  const int* table = a.page_table + (size_t)seq * a.pt_stride;
  const int last = pos0 + n - 1;

  auto lowest = [&](int pos) {
    return a.window > 0 ? (a.mask_mode == 1 ? pos / a.window * a.window : max(0, pos - a.window + 1)) : 0;
  };
  const int lo = lowest(pos0);  // (the first token sees the furthest back)
  const int nfront = (min(a.keep_first, lo) + TILE_KEYS - 1) / TILE_KEYS;  // tiles of kept keys in front of the window
  const int first = max(nfront, lo / TILE_KEYS), ntiles = nfront + last / TILE_KEYS - first + 1;
  auto tile_start = [&](int i) { return (i < nfront ? i : first + i - nfront) * TILE_KEYS; };

  __syncthreads();  // (a block of several groups of heads: the last one's reads are done)
  for (int i = tid; i < R * (D / 4); i += NT) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    const bool there = r < rows;
    const T* src = (const T*)a.q;
    if (there) src += (size_t)(t0 + r / gn) * a.q_stride + (size_t)(kvh * G + g0 + r % gn) * D + d;
    bring4(qs + r * LK + d, src, there);
  }
  // Where the keys of tile i lie: thread j < TILE_KEYS asks the page table for key j (`find`) and writes the answer
  // down for all (`note`), a tile ahead, so that nobody waits for the table between the tiles.
  auto find = [&](int i) -> long {
    const int key = tile_start(i) + tid;
    if (tid >= TILE_KEYS || key > last) return -1;
    const int page = table[key / a.page_size];
    if (page >= 0 && page < a.num_pages) return ((long)page * a.KVH + kvh) * a.page_size + key % a.page_size;
    // a page the window has passed is gone from the table; one that some token still sees must be there
    if (key >= lo || key < a.keep_first) atomicOr(a.err, DSP_ERR_BAD_PAGE);
    return -1;
  };
  auto note = [&](int i, long at) {
    if (tid < TILE_KEYS) slot[(i & 1) * TILE_KEYS + tid] = at;
  };
  // a warp copies whole rows, a lane 16 bytes (8 of bfloat16) of each
  const int lane = tid & 31, warp = tid >> 5;
  auto bring = [&](int i, const T* pool, int width, float* to, int ld) {
    if (lane < width / 4) {
#pragma unroll 2
      for (int j = warp; j < TILE_KEYS; j += NT / 32) {
        const long at = slot[(i & 1) * TILE_KEYS + j];
        bring4(to + j * ld + lane * 4, at >= 0 ? pool + at * width + lane * 4 : pool, at >= 0);
      }
    }
    end_group();
  };
  auto bring_keys = [&](int i) { bring(i, (const T*)a.k_pool, D, ks, LK); };
  auto bring_values = [&](int i) { bring(i, (const T*)a.v_pool, Dv, vs, LV); };

  float m[RI], l[RI], acc[RI][4 * DJ];
  int pos[RI], low[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = ty + i * TY;
    pos[i] = r < rows ? pos0 + r / gn : -1;
    low[i] = r < rows ? lowest(pos[i]) : 0;
    m[i] = a.sink ? ((a.sink_values && r < rows) ? a.sink_values[kvh * G + g0 + r % gn] : 0.f) : -INFINITY;
    l[i] = a.sink ? 1.f : 0.f;
#pragma unroll
    for (int d = 0; d < 4 * DJ; ++d) acc[i][d] = 0.f;
  }
  note(0, find(0));
  __syncthreads();
  bring_keys(0);
  bring_values(0);
  for (int t = 0; t < ntiles; ++t) {
    const int kt = tile_start(t);
    const long next = t + 1 < ntiles ? find(t + 1) : -1;
    wait_groups<1>();
    __syncthreads();
    float s[RI][KJ];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
      for (int j = 0; j < KJ; ++j) s[i][j] = 0.f;
#pragma unroll 2
    for (int d = 0; d < D; d += 4) {
      float4 x[RI];
#pragma unroll
      for (int i = 0; i < RI; ++i) x[i] = *reinterpret_cast<const float4*>(qs + (ty + i * TY) * LK + d);
      float4 y[KJ];
#pragma unroll
      for (int j = 0; j < KJ; ++j) y[j] = *reinterpret_cast<const float4*>(ks + (tx + j * TX) * LK + d);
      // dimension after dimension over all sums: neighbouring instructions do not wait for one another
#pragma unroll
      for (int j = 0; j < KJ; ++j)
#pragma unroll
        for (int i = 0; i < RI; ++i) s[i][j] = fmaf(x[i].x, y[j].x, s[i][j]);
#pragma unroll
      for (int j = 0; j < KJ; ++j)
#pragma unroll
        for (int i = 0; i < RI; ++i) s[i][j] = fmaf(x[i].y, y[j].y, s[i][j]);
#pragma unroll
      for (int j = 0; j < KJ; ++j)
#pragma unroll
        for (int i = 0; i < RI; ++i) s[i][j] = fmaf(x[i].z, y[j].z, s[i][j]);
#pragma unroll
      for (int j = 0; j < KJ; ++j)
#pragma unroll
        for (int i = 0; i < RI; ++i) s[i][j] = fmaf(x[i].w, y[j].w, s[i][j]);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      float top = -INFINITY;
      unsigned hidden = 0;  // bit j: key j is not this row's
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const int key = kt + tx + j * TX;
        const bool seen = key <= pos[i] && (key >= low[i] || key < a.keep_first) && slot[(t & 1) * TILE_KEYS + tx + j * TX] >= 0;
        s[i][j] = seen ? s[i][j] * a.scale : -INFINITY;
        hidden |= (seen ? 0u : 1u) << j;
        top = fmaxf(top, s[i][j]);
      }
#pragma unroll
      for (int o = TX / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float m_new = fmaxf(m[i], top);
      // m_new stays -inf for rows that have seen no key yet
      const float alpha = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);
      // a hidden key's weight is -0, which no seen key's is: below it is told from a weight that is merely small
      float p[KJ];
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        p[j] = s[i][j] == -INFINITY ? ((hidden >> j & 1u) ? -0.f : 0.f) : expf(s[i][j] - m_new);
        ps[(ty + i * TY) * LP + tx + j * TX] = p[j];
      }
      // keys l, l + 32 first, then their neighbours 16, 8, 4, 2 and 1 away, on either grid of threads: a token's sum is
      // the same alone and among the others of a portion
      float sum;
      static_assert(KJ == 2 || KJ == 4, "32 or 16 threads a row");
      if constexpr (KJ == 2) sum = p[0] + p[1];
      else sum = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
      for (int o = TX / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      m[i] = m_new;
      l[i] = l[i] * alpha + sum;
#pragma unroll
      for (int d = 0; d < 4 * DJ; ++d) acc[i][d] *= alpha;
    }
    note(t + 1, next);  // (the slots of tile t - 1, which all have left)
    __syncthreads();  // the keys have been read
    if (t + 1 < ntiles) bring_keys(t + 1); else end_group();
    wait_groups<1>();
    __syncthreads();  // the values are there (and every row of ps)
    // where some row does not see every key, a key that a row does not see (weight -0) must not reach it: 0 times a
    // value that is no number is none either
    const bool all_seen = kt + TILE_KEYS - 1 <= pos0 && kt >= lowest(last);
    auto add_values = [&](auto some_hidden) {
#pragma unroll 2
      for (int j = 0; j < TILE_KEYS; j += 4) {
        float p[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(ps + (ty + i * TY) * LP + j);
          p[i][0] = v.x, p[i][1] = v.y, p[i][2] = v.z, p[i][3] = v.w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int dj = 0; dj < DJ; ++dj) {
            const int d = (tx + dj * TX) * 4;
            if (d >= Dv) continue;
            const float4 v = *reinterpret_cast<const float4*>(vs + (j + e) * LV + d);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
              if (decltype(some_hidden)::value && __float_as_uint(p[i][e]) == 0x80000000u) continue;
              acc[i][4 * dj] = fmaf(p[i][e], v.x, acc[i][4 * dj]);
              acc[i][4 * dj + 1] = fmaf(p[i][e], v.y, acc[i][4 * dj + 1]);
              acc[i][4 * dj + 2] = fmaf(p[i][e], v.z, acc[i][4 * dj + 2]);
              acc[i][4 * dj + 3] = fmaf(p[i][e], v.w, acc[i][4 * dj + 3]);
            }
          }
      }
    };
    if (all_seen) add_values(std::false_type{}); else add_values(std::true_type{});
    __syncthreads();  // the values have been read
    if (t + 1 < ntiles) bring_values(t + 1); else end_group();
  }
  wait_groups<0>();
  float* os = ks;  // [R][Dv] results before they are turned back (with turn_freq)
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = ty + i * TY;
    if (r >= rows) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const int tok = t0 + r / gn;
#pragma unroll
    for (int dj = 0; dj < DJ; ++dj)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = (tx + dj * TX) * 4 + e;
        if (d >= Dv) continue;
        const size_t col = (size_t)(kvh * G + g0 + r % gn) * Dv + d;
        float y = acc[i][4 * dj + e] * inv;
        if (a.gate) y /= 1.f + expf(-a.gate[(size_t)tok * a.ldg + col]);
        if (a.turn_freq)
          os[r * Dv + d] = y;
        else
          st_any(a.out, a.out_dtype, (size_t)tok * a.out_stride + col, y);
      }
  }
  if (a.turn_freq) {
    __syncthreads();
    const int half = Dv / 2;
    for (int i = tid; i < rows * Dv; i += NT) {
      const int r = i / Dv, d = i % Dv, mth = d < half ? d : d - half;
      float sn, cn;
      sincosf((float)(pos0 + r / gn) * a.turn_freq[mth], &sn, &cn);
      // the inverse turn: (u, v) -> (u cos + v sin, v cos - u sin)
      const float y = d < half ? os[i] * cn + os[i + half] * sn : os[i] * cn - os[i - half] * sn;
      st_any(a.out, a.out_dtype, (size_t)(t0 + r / gn) * a.out_stride + (size_t)(kvh * G + g0 + r % gn) * Dv + d, y);
    }
  }
}

constexpr int FEW_ROWS = 8;

template <typename T, int ROWS, int NT>
__global__ void __launch_bounds__(NT) attn_rows_kernel(const RowsArgs a) {
  extern __shared__ __align__(16) float rows_smem[];
  const int t0 = (int)gridDim.x - 1 - (int)blockIdx.x, kvh = blockIdx.y, pos0 = a.positions[t0];  // the longest first
  if (pos0 < 0) return;
  const int seq = a.seq_of_token[t0], G = a.H / a.KVH, per = max(1, ROWS / G);
  if (pos0 % per && t0 > 0 && a.seq_of_token[t0 - 1] == seq && a.positions[t0 - 1] == pos0 - 1) return;  // inside a run
  int n = 1;
  while (n < per && (pos0 + n) % per && t0 + n < a.T && a.seq_of_token[t0 + n] == seq && a.positions[t0 + n] == pos0 + n) ++n;
  if (n * G <= FEW_ROWS)
    attn_rows<T, FEW_ROWS, NT / 32, NT>(a, rows_smem, t0, n, pos0, seq, kvh, 0, G);
  else
    for (int g0 = 0; g0 < G; g0 += ROWS) attn_rows<T, ROWS, NT / 16, NT>(a, rows_smem, t0, n, pos0, seq, kvh, g0, min(ROWS, G - g0));
}

template <typename T, int ROWS, int NT>
int launch_rows(const RowsArgs& a, cudaStream_t stream) {
  const size_t smem = (size_t)((ROWS + TILE_KEYS) * (a.D + 4) + TILE_KEYS * (a.Dv + 4) + ROWS * (TILE_KEYS + 4)) * sizeof(float) +
                      2 * TILE_KEYS * sizeof(long);
  DSP_CUDA(cudaFuncSetAttribute(attn_rows_kernel<T, ROWS, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  attn_rows_kernel<T, ROWS, NT><<<dim3(a.T, a.KVH), NT, smem, stream>>>(a);
  DSP_CHECK_LAUNCH("dsp_attn_generic");
  return 0;
}
// Rows of a run and threads of a block, by the blocks that a step gives: `singles` single tokens, portions of the other
// tokens, `longest` the tokens of its longest context (0: not known).  The bits are the same.  A block's time is that of its
// tiles, one after the other, and a portion that begins a prompt has half as many as its last block has: runs of 16 rows
// while the step takes no longer than its longest block (two of them on an SM), for heads of which a group fills no more;
// many single tokens of up to 8 rows share the SMs better with 128 threads, and so do many blocks of up to 96 dimensions,
// of which three fit an SM then.  us with 16 rows and 256 threads / 32 and 256 / 32 and 128: 12 heads of 128 on 2, 264 tokens
// behind 600 keys 154 / 200 / 211, 400 behind 600 263 / 236 / 242, 500 alone 95 / 120 / 126; 40 on 2, 128 behind 600 267 / 179 /
// 183; 16 heads of 64 on 8, 800 behind 600 370 / 368 / 295; single tokens at 600 keys, 32 heads of 128 on 8, 64 of them 145 /
// 143 / 133, one 49 / 48 / 55.
enum { RUNS_16 = 0, RUNS_32 = 1, RUNS_32_NARROW = 2 };
int rows_kernel(int T, int singles, int longest, int H, int KVH, int D, int Dv, int sms) {
  const int G = H / KVH, rest = T - singles;
  const double share = longest > 0 ? 1.0 - 0.5 * (rest < longest ? rest : longest) / longest : 1.0;  // of a portion's block
  auto blocks = [&](int rows) {
    const int per = G < rows ? rows / G : 1;
    return KVH * (singles + share * ((rest + per - 1) / per));
  };
  const double alone = (double)KVH * singles, runs = blocks(32);
  if (G <= FEW_ROWS && alone > sms && 2.0 * alone >= runs) return RUNS_32_NARROW;
  if (G <= 16 && (rest == 0 || blocks(16) <= 2.0 * sms)) return RUNS_16;
  return runs > 1.9 * sms && D + Dv <= 192 ? RUNS_32_NARROW : RUNS_32;
}
template <typename T>
int launch_rows(const RowsArgs& a, int singles, int longest, cudaStream_t stream) {
  const int sms = dsp_num_sms();
  switch (rows_kernel(a.T, singles, longest, a.H, a.KVH, a.D, a.Dv, sms > 0 ? sms : 148)) {
    case RUNS_16: return launch_rows<T, 16, 256>(a, stream);
    case RUNS_32: return launch_rows<T, 32, 256>(a, stream);
    default: return launch_rows<T, 32, 128>(a, stream);
  }
}

// Whether rows of `width` elements at `stride` from `p` consist of whole pieces of four elements.
bool whole_pieces(const void* p, long stride, int width, int dtype) {
  return (uintptr_t)p % (dtype == DSP_F32 ? 16 : 8) == 0 && stride % 4 == 0 && width % 4 == 0;
}
}  // namespace

// Which kernel runs (0: runs of 16 rows, 1: of 32, 2: of 32 on 128 threads).
extern "C" int dsp_attn_rows_choice(int T, int singles, int longest, int H, int KVH, int D, int Dv, int sms) {
  return rows_kernel(T, singles, longest, H, KVH, D, Dv, sms);
}

// singles: of the T tokens, so many are the only ones of their request; longest: tokens of the longest context (0: not
// known).  They decide how the work is cut.
extern "C" int dsp_attn_generic(const void* q, long q_stride, const void* k_pool,
                                const void* v_pool, const int* page_table, int pt_stride,
                                const int* positions, const int* seq_of_token, void* out,
                                long out_stride, int T, int singles, int longest, int H, int KVH, int D, int Dv, int page_size,
                                int num_pages, int window, int mask_mode, int keep_first, float scale,
                                int sink, const float* sink_values, const float* turn_freq, const float* gate, long ldg, int dtype, int out_dtype,
                                cudaStream_t stream) {
  if (T == 0) return 0;
  DSP_REQUIRE(KVH > 0 && H % KVH == 0, "dsp_attn_generic: H=%d is not a multiple of KVH=%d", H, KVH);
  DSP_REQUIRE(D > 0 && Dv > 0 && Dv <= THREADS * DPT && D <= 4096,
              "dsp_attn_generic: key size %d or value size %d outside the kernel's range (values up to %d)", D, Dv,
              THREADS * DPT);
  DSP_REQUIRE(KVH <= 65535, "dsp_attn_generic: too many KV heads");
  DSP_REQUIRE(mask_mode == 0 || mask_mode == 1, "dsp_attn_generic: unknown mask mode %d", mask_mode);
  DSP_REQUIRE(keep_first >= 0, "dsp_attn_generic: keep_first=%d", keep_first);
  DSP_REQUIRE(!gate || !turn_freq, "dsp_attn_generic: results are gated or turned back, not both");
  DSP_REQUIRE(!turn_freq || Dv % 2 == 0, "dsp_attn_generic: values of an odd width %d cannot be turned", Dv);
  DSP_REQUIRE(singles >= 0 && singles <= T, "dsp_attn_generic: %d single tokens of %d", singles, T);
  int* err = dsp_device_error_ptr();
  DSP_REQUIRE(err != nullptr, "dsp_attn_generic: no device error word");
  if ((dtype == DSP_F32 || dtype == DSP_BF16) && D <= MAX_DIM && Dv <= MAX_DIM && whole_pieces(q, q_stride, D, dtype) &&
      whole_pieces(k_pool, 0, D, dtype) && whole_pieces(v_pool, 0, Dv, dtype)) {
    const RowsArgs a = {q, k_pool, v_pool, page_table, positions, seq_of_token, out, sink_values, turn_freq, gate,
                        q_stride, out_stride, ldg, pt_stride, T, H, KVH, D, Dv, page_size, num_pages, window, mask_mode,
                        keep_first, sink, out_dtype, scale, err};
    return dtype == DSP_F32 ? launch_rows<float>(a, singles, longest, stream) : launch_rows<bf16>(a, singles, longest, stream);
  }
  const size_t smem = (size_t)(GCHUNK * D + GCHUNK * THREADS + (turn_freq ? GCHUNK * Dv : 0)) * sizeof(float) +
                      THREADS * sizeof(long);
  dim3 grid(T, KVH);
  if (dtype == DSP_F32) {
    static size_t configured = 0;
    if (smem > configured) {
      DSP_CUDA(cudaFuncSetAttribute(attn_generic_kernel<float>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      configured = smem;
    }
    attn_generic_kernel<float><<<grid, THREADS, smem, stream>>>(
        (const float*)q, q_stride, (const float*)k_pool, (const float*)v_pool, page_table, pt_stride,
        positions, seq_of_token, out, out_dtype, out_stride, H, KVH, D, Dv, page_size, num_pages, window,
        mask_mode, keep_first, scale, sink, sink_values, turn_freq, gate, ldg, err);
  } else if (dtype == DSP_BF16) {
    static size_t configured = 0;
    if (smem > configured) {
      DSP_CUDA(cudaFuncSetAttribute(attn_generic_kernel<bf16>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      configured = smem;
    }
    attn_generic_kernel<bf16><<<grid, THREADS, smem, stream>>>(
        (const bf16*)q, q_stride, (const bf16*)k_pool, (const bf16*)v_pool, page_table, pt_stride,
        positions, seq_of_token, out, out_dtype, out_stride, H, KVH, D, Dv, page_size, num_pages, window,
        mask_mode, keep_first, scale, sink, sink_values, turn_freq, gate, ldg, err);
  } else {
    DSP_REQUIRE(false, "dsp_attn_generic: unknown dtype %d", dtype);
  }
  DSP_CHECK_LAUNCH("dsp_attn_generic");
  return 0;
}
