// The layers of a dense decoder behind one call: for every layer
//
//   qkv = norm1(x) Wqkv^T + b;  rotation, keys and values into the pages;  attention;
//   x += attention Wo^T (+ b);  x += (act(norm2(x) Wg^T) * norm2(x) Wu^T) Wd^T
//
// Host code only: it calls the entry points of this library in the order, with the choices and with the
// arguments with which the parts call them one by one, so the results have the same bits.  A step that is not
// replayed from a graph launches some 230 kernels; called from Python each took the host 17 us (an output tensor,
// checks, twenty converted arguments, the call), more than many of them take the device: 3.9 ms for a prompt of
// 137 tokens of which the device was busy 2.1.
#include "common.cuh"

extern "C" {
int dsp_rmsnorm(void* x, const void* delta, const void* w, void* y, const int* rows, int n_rows, int hidden, float eps,
                int write_back, int dtype, cudaStream_t stream);
int dsp_rope_kv_store(void* qkv, const int* positions, const int* seq_of_token, const int* page_table, int pt_stride,
                      void* k_pool, void* v_pool, const float* inv_freq, int T, int H, int KVH, int D, int rotary_dim,
                      int page_size, int num_pages, int write_kv, int early, int dtype, cudaStream_t stream);
int dsp_gemm_stream(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                    long ldc, int M, int N, int K, int out_dtype, int target_ctas, int epilogue, long late_trigger_bytes,
                    const void* norm_src, long ld_src, float norm_eps, const void* gain2, void* C2, long ldc2,
                    cudaStream_t stream);
int dsp_gemm_tcgen05(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C,
                     long ldc, int M, int N, int K, int out_dtype, int pair_mode, int epilogue, cudaStream_t stream);
int dsp_gemm_few_rows_faster(int M, int N, int K, int target_ctas);
int dsp_gemm_pairs(const void* A, long lda, const void* W, const void* bias, const void* residual, long ldr, void* C, long ldc,
                   int M, int N, int K, int out_dtype, int epilogue, const float* act, int splits, int chunks, cudaStream_t stream);
int dsp_gemm_pairs_faster(int M, int N, int K, int target_ctas, int result);
int dsp_attn_combine(const float* part_o, const float* part_ml, void* out, long out_stride, int num_tokens, int H, int D,
                     int splits, int dtype, cudaStream_t stream);
}

namespace {
// The attention entry points live in libraries of their own (one per head size).
typedef int (*AttnMma)(const void*, long, const void*, const void*, const int*, int, const int*, const int*, const int*,
                       const int*, int, int, void*, long, float*, float*, int, int, int, int, int, int, int, int, int,
                       int, float, const float*, int, int, int, int*, cudaStream_t);
typedef int (*AttnTcgen05)(const void*, long, const void*, const void*, const int*, int, const int*, const int*,
                           const int*, const int*, int, int, void*, long, int, int, int, int, int, int, float, int*,
                           cudaStream_t);
}  // namespace

// Both structures are filled by ops/dense_chain.py: eight bytes a field, in this order.
struct DspDenseLayer {
  const void *w_qkv, *b_qkv, *w_o, *b_o, *w_gate_up, *w_down, *norm1, *norm2;
  void *k_pool, *v_pool;
  const int* page_table;
  const float* inv_freq;
  long pt_stride, num_pages, window, write_kv;
  double eps1, eps2, scale;
};
struct DspDenseStep {
  long layers, T, singles;  // rows of the flat batch; single tokens, which come first
  long hidden, H, KVH, D, inter, rotary_dim, page_size, epilogue;
  const int *positions, *seq_of_token, *q_start, *ctx_len;
  // tiles of 64 query rows (single tokens first) and of 128 (null: portions run on the tiles of 64)
  const int *tile_seq, *tile_tok0, *big_seq, *big_tok0;
  long tiles, big_tiles, per_tile, per_big_tile;
  long splits, outer;  // of a single token's keys: inside a cluster, beyond it
  float *part_o, *part_ml;
  long fused_rope;  // the single tokens' kernel rotates and stores their keys itself
  void *x, *h, *qkv, *heads, *act, *scaled_a, *scaled_b;  // scaled_*: null above the rows a norm is split over products
  long target_ctas, always_few, late_trigger_bytes;       // as ops/gemm.py passes them
  void *attn_mma, *attn_tcgen05;
  int* err;
  void* stream;
};

extern "C" int dsp_dense_layers(const DspDenseStep* step, const DspDenseLayer* layers, long* launches) {
  const DspDenseStep& s = *step;
  const cudaStream_t stream = (cudaStream_t)s.stream;
  const int T = (int)s.T, n1 = (int)s.singles, hidden = (int)s.hidden, inter = (int)s.inter;
  const int H = (int)s.H, KVH = (int)s.KVH, D = (int)s.D, wide = (H + 2 * KVH) * D;
  long count = 0;
  if (T == 0) return 0;
#define DSP_STEP(call)          \
  do {                          \
    const int rc__ = (call);    \
    if (rc__ != 0) return rc__; \
    ++count;                    \
  } while (0)

  // The kernel of a product, asked once for each of the layers' sizes (an answer takes the host about two microseconds).
  // The one on CTA pairs reads four biases at a time: a bias that does not begin on eight bytes goes to the others.
  enum { MANY = 0, FEW = 1, PAIRS = 2 };
  struct { int N, K, kernel; bool fours; } chosen[8];
  int num_chosen = 0;
  auto choose = [&](int N, int K, const void* bias) -> int {
    if (T <= s.always_few) return FEW;
    const bool fours = ((uintptr_t)bias & 7) == 0;
    for (int i = 0; i < num_chosen; ++i)
      if (chosen[i].N == N && chosen[i].K == K && chosen[i].fours == fours) return chosen[i].kernel;
    int kernel = fours ? dsp_gemm_pairs_faster(T, N, K, (int)s.target_ctas, 0) : 0;
    if (kernel == 1) kernel = PAIRS;
    else if (kernel == 0) kernel = dsp_gemm_few_rows_faster(T, N, K, (int)s.target_ctas);
    if (kernel >= 0 && num_chosen < 8) chosen[num_chosen++] = {N, K, kernel, fours};
    return kernel;
  };
  // C = A W^T (+ bias) (+ C): the kernel that ops/gemm.py chooses.  `scaled`, `eps`: A is x under a norm still to be
  // applied, `scaled` those rows times its gain.  `gain`, `scaled_out`: the norm after this product, where its kernel
  // can prepare it; *prepared says whether it did.
  auto product = [&](const void* A, int K, const void* W, int N, const void* bias, bool add, void* C, const void* scaled,
                     float eps, const void* gain, void* scaled_out, bool* prepared) -> int {
    const void* residual = add ? C : nullptr;
    if (prepared) *prepared = false;
    const int kernel = choose(N, K, bias);
    if (kernel < 0) return kernel;
    if (kernel == PAIRS) return dsp_gemm_pairs(A, K, W, bias, residual, add ? N : 0, C, N, T, N, K, DSP_BF16, 0, nullptr, 0, 0, stream);
    if (kernel == FEW) {
      const bool prepare = gain && scaled_out;
      if (prepared) *prepared = prepare;
      return dsp_gemm_stream(scaled ? scaled : A, K, W, bias, residual, add ? N : 0, C, N, T, N, K, DSP_BF16,
                             (int)s.target_ctas, 0, s.late_trigger_bytes, scaled ? s.x : nullptr, scaled ? K : 0,
                             scaled ? eps : 0.f, prepare ? gain : nullptr, prepare ? scaled_out : nullptr,
                             prepare ? N : 0, stream);
    }
    return dsp_gemm_tcgen05(A, K, W, bias, residual, add ? N : 0, C, N, T, N, K, DSP_BF16, 1, 0, stream);
  };

  const int pairs_gate_up = T > s.always_few ? dsp_gemm_pairs_faster(T, 2 * inter, hidden, (int)s.target_ctas, 2) : 0;
  if (pairs_gate_up < 0) return pairs_gate_up;
  bool ready = false;  // scaled_b holds x times the next norm1's gain
  for (long i = 0; i < s.layers; ++i) {
    const DspDenseLayer& l = layers[i];
    if (!ready) DSP_STEP(dsp_rmsnorm(s.x, nullptr, l.norm1, s.h, nullptr, T, hidden, (float)l.eps1, 0, DSP_BF16, stream));
    DSP_STEP(product(s.h, hidden, l.w_qkv, wide, l.b_qkv, false, s.qkv, ready ? s.scaled_b : nullptr, (float)l.eps1,
                     nullptr, nullptr, nullptr));
    const int first = s.fused_rope ? n1 : 0;
    if (T > first)
      DSP_STEP(dsp_rope_kv_store((bf16*)s.qkv + (size_t)first * wide, s.positions + first, s.seq_of_token + first,
                                 l.page_table, (int)l.pt_stride, l.write_kv ? l.k_pool : nullptr,
                                 l.write_kv ? l.v_pool : nullptr, l.inv_freq, T - first, H, KVH, D, (int)s.rotary_dim,
                                 l.write_kv ? (int)s.page_size : 1, l.write_kv ? (int)l.num_pages : 0, (int)l.write_kv, 1,
                                 DSP_BF16, stream));
    auto mma = [&](int offset, int tiles, int splits, bool single) -> int {
      const bool fused = single && s.fused_rope, ranges = single && s.outer > 1;
      const int rc = ((AttnMma)s.attn_mma)(
          s.qkv, wide, l.k_pool, l.v_pool, l.page_table, (int)l.pt_stride, s.q_start, s.ctx_len, s.tile_seq, s.tile_tok0,
          offset, tiles, s.heads, (long)H * D, ranges ? s.part_o : nullptr, ranges ? s.part_ml : nullptr, H, KVH,
          (int)s.per_tile, (int)s.page_size, (int)l.num_pages, (int)l.window, splits, splits > 1 ? 1 : 0, single ? 1 : 0,
          single ? (int)s.outer : 1, (float)l.scale, fused ? l.inv_freq : nullptr, fused ? (int)s.rotary_dim : 0,
          fused ? 1 : 0, fused ? (int)l.write_kv : 0, s.err, stream);
      if (rc != 0) dsp_set_error("dsp_dense_layers: the attention over tiles of 64 rows answered %d", rc);
      return rc;
    };
    if (n1 > 0) {
      DSP_STEP(mma(0, n1, (int)s.splits, true));
      if (s.outer > 1)
        DSP_STEP(dsp_attn_combine(s.part_o, s.part_ml, s.heads, (long)H * D, n1, H, D, (int)s.outer, DSP_BF16, stream));
    }
    if (s.big_seq != nullptr) {
      if (s.big_tiles > n1) {
        const int rc = ((AttnTcgen05)s.attn_tcgen05)(
            s.qkv, wide, l.k_pool, l.v_pool, l.page_table, (int)l.pt_stride, s.q_start, s.ctx_len, s.big_seq, s.big_tok0,
            n1, (int)s.big_tiles - n1, s.heads, (long)H * D, H, KVH, (int)s.per_big_tile, (int)s.page_size,
            (int)l.num_pages, (int)l.window, (float)l.scale, s.err, stream);
        if (rc != 0) dsp_set_error("dsp_dense_layers: the attention over tiles of 128 rows answered %d", rc);
        DSP_STEP(rc);
      }
    } else if (s.tiles > n1) {
      DSP_STEP(mma(n1, (int)s.tiles - n1, 1, false));
    }
    bool normed = false;
    DSP_STEP(product(s.heads, H * D, l.w_o, hidden, l.b_o, true, s.x, nullptr, 0.f, l.norm2, s.scaled_a, &normed));
    if (!normed) DSP_STEP(dsp_rmsnorm(s.x, nullptr, l.norm2, s.h, nullptr, T, hidden, (float)l.eps2, 0, DSP_BF16, stream));
    if (T <= s.always_few)
      DSP_STEP(dsp_gemm_stream(normed ? s.scaled_a : s.h, hidden, l.w_gate_up, nullptr, nullptr, 0, s.act, inter, T,
                               2 * inter, hidden, DSP_BF16, (int)s.target_ctas, (int)s.epilogue, s.late_trigger_bytes,
                               normed ? s.x : nullptr, normed ? hidden : 0, normed ? (float)l.eps2 : 0.f, nullptr, nullptr,
                               0, stream));
    else if (pairs_gate_up)
      DSP_STEP(dsp_gemm_pairs(s.h, hidden, l.w_gate_up, nullptr, nullptr, 0, s.act, inter, T, 2 * inter, hidden, DSP_BF16,
                              (int)s.epilogue, nullptr, 0, 0, stream));
    else
      DSP_STEP(dsp_gemm_tcgen05(s.h, hidden, l.w_gate_up, nullptr, nullptr, 0, s.act, inter, T, 2 * inter, hidden,
                                DSP_BF16, 1, (int)s.epilogue, stream));
    const bool more = i + 1 < s.layers;
    DSP_STEP(product(s.act, inter, l.w_down, hidden, nullptr, true, s.x, nullptr, 0.f, more ? layers[i + 1].norm1 : nullptr,
                     s.scaled_b, &ready));
  }
#undef DSP_STEP
  *launches = count;
  return 0;
}
