"""The layers of a dense decoder behind one call of the kernel library (``csrc/dense_chain.cu``).

A model whose layers are all ``pre_norm`` blocks of ``gqa_attention`` and ``swiglu`` under ``rms_norm`` runs
them through ``run_layers``: the same kernels in the same order as its parts would launch, called from C.
``plan`` looks at the assembled parts once; every address is read from the parts, the cache and the step
when a step runs."""
from __future__ import annotations

import ctypes
import struct

import torch

from dispec_b200.ops import attention as attn_ops
from dispec_b200.ops import gemm
from dispec_b200.ops import library as L
from dispec_b200.ops import tuning

_LAYER = struct.Struct("12q4q3d")
_STEP = struct.Struct("11q4q4q4q2q2q1q7q3q2q1q1q")


def plan(model) -> bool:
    """Whether every layer run of ``model`` is of the kind above, with the same sizes."""
    from dispec_b200.parts.attention import GQAAttention
    from dispec_b200.parts.block import PreNormBlock
    from dispec_b200.parts.embedding import TokenEmbedding
    from dispec_b200.parts.norms import RMSNorm
    from dispec_b200.parts.rotary import RotaryEncoding
    from dispec_b200.parts.swiglu import SwiGLUFeedForward

    if model.dtype != torch.bfloat16 or type(model.embedding) is not TokenEmbedding or not model.schedule:
        return False
    sizes = set()
    for call, state in zip(model.schedule, model.call_state):
        block = model.layers[call.layer]
        if type(block) is not PreNormBlock or call.entry is not None or state is not None:
            return False
        mixer, ff, norms = block.mixer, block.feed_forward, (block.mixer_norm, block.ffn_norm)
        if (type(mixer) is not GQAAttention or type(ff) is not SwiGLUFeedForward or any(type(n) is not RMSNorm for n in norms)
                or type(mixer.position_encoding) is not RotaryEncoding or ff.out_float32 or ff.block != gemm.SWIGLU_BLOCK):
            return False
        rot = mixer.position_encoding.rotation()
        if rot is None or rot.layout != "halves" or rot.magnitude != 1.0 or not rot.rotary_dim:
            return False
        sizes.add((mixer.hidden_size, mixer.num_heads, mixer.num_kv_heads, mixer.head_dim, rot.rotary_dim,
                   ff.intermediate_size, ff.act))
    if len(sizes) != 1:
        return False
    hidden, H, KVH, D, _, inter, _ = sizes.pop()
    # rows of whole 16-byte pieces everywhere, heads that the tensor-core kernels take
    return (hidden % 8 == 0 and H * D % 8 == 0 and inter % 8 == 0 and KVH * D % 8 == 0
            and H // KVH <= attn_ops.DECODE_KERNEL_MAX_GROUP
            and attn_ops.tensor_core_supported(D, H // KVH, torch.bfloat16))


def run_layers(model, ctx, x: torch.Tensor) -> bool:
    """Runs the layers on the rows ``x`` in place; False (nothing has run) where this step is not for it.  A step that
    is being captured is not: its launches are replayed from the graph, whoever made them, and one row a step was
    1.5 % slower on this function's buffers (950 us against 935) than on those of the parts."""
    if ctx.graph_capture:
        return False
    block = model.layers[model.schedule[0].layer]
    mixer, ff = block.mixer, block.feed_forward
    H, KVH, D, hidden, inter = (mixer.num_heads, mixer.num_kv_heads, mixer.head_dim, mixer.hidden_size,
                                ff.intermediate_size)
    group, T, n_dec, dev = H // KVH, x.shape[0], ctx.num_decode_seqs, x.device
    tpt = attn_ops.tokens_per_tile(group)
    splits = ctx.decode_splits or attn_ops.choose_splits(n_dec, KVH, ctx.max_ctx_len, dev)
    if T == 0 or tpt not in ctx.attention_tiles or splits > tuning.CLUSTER_MAX_SPLITS:
        return False
    outer = ctx.decode_outer or attn_ops.choose_outer(n_dec, KVH, ctx.max_ctx_len, splits, dev)
    tile_seq, tile_tok0, num_tiles = ctx.attention_tiles[tpt]
    big = attn_ops.prefill_tokens_per_tile(group)
    big_seq = big_tok0 = None
    big_tiles, tcgen05 = 0, 0
    if big in ctx.attention_tiles and attn_ops.tcgen05_supported(D, group, ctx.page_size, torch.bfloat16):
        big_seq, big_tok0, big_tiles = ctx.attention_tiles[big]
        if big_tiles > n_dec:
            tcgen05 = L.address_of(L.prefill_attention_library(D), f"dsp_attn_tcgen05_d{D}")
    mma = L.address_of(L.attention_library(D), f"dsp_attn_mma_d{D}")
    part_o = part_ml = None
    if n_dec and outer > 1:
        part_o, part_ml = attn_ops._partial_buffers(dev, n_dec * H, outer, D)
    rotary_dim = mixer.position_encoding.rotation().rotary_dim
    fused = attn_ops.decode_rope_fusable(ctx, H, KVH, D, rotary_dim, x.dtype)

    new = lambda columns: torch.empty((T, columns), dtype=x.dtype, device=dev)
    # normed rows are dead when attention writes its heads, the q/k/v rows when the feed-forward writes its units:
    # two buffers for the four keep more of a long portion in the L2
    h = heads = new(max(hidden, H * D))
    qkv = act = new(max((H + 2 * KVH) * D, inter))
    scaled_a = scaled_b = None
    if T <= gemm.NORM_SPLIT_MAX_ROWS:  # norms are split over the products around them
        scaled_a, scaled_b = new(hidden), new(hidden)

    address = lambda t: t.data_ptr() if t is not None else 0
    table = bytearray(_LAYER.size * len(model.schedule))
    for i, call in enumerate(model.schedule):
        b = model.layers[call.layer]
        m, f = b.mixer, b.feed_forward
        cache = ctx.cache_view(model.placement[model.call_cache[i]], call.write)
        rot = m.position_encoding.rotation()
        keys, values = cache.key_pool, cache.value_pool
        # weights are kept as a source handed them over; where one begins off a 16-byte address, its product is one that
        # the parts choose
        if (m.w_qkv.data_ptr() | m.w_o.data_ptr() | f.w_gate_up.data_ptr() | f.w_down.data_ptr()) % 16:
            return False
        _LAYER.pack_into(table, i * _LAYER.size, address(m.w_qkv), address(m.b_qkv), address(m.w_o), address(m.b_o),
                         address(f.w_gate_up), address(f.w_down), address(b.mixer_norm.weight),
                         address(b.ffn_norm.weight), address(keys), address(values), address(cache.page_table),
                         address(rot.inv_freq), cache.page_table.stride(0), cache.num_pages, m.window,
                         int(cache.write), b.mixer_norm.eps, b.ffn_norm.eps,
                         m.scale * m.position_encoding.score_scale())
    step = _STEP.pack(
        len(model.schedule), T, n_dec, hidden, H, KVH, D, inter, rotary_dim, ctx.page_size,
        gemm.EPI_SWIGLU if ff.act == "silu" else gemm.EPI_GEGLU,
        address(ctx.positions), address(ctx.seq_of_token), address(ctx.q_start), address(ctx.ctx_len),
        address(tile_seq), address(tile_tok0), address(big_seq), address(big_tok0), num_tiles, big_tiles, tpt, big,
        splits, outer, address(part_o), address(part_ml), int(fused), address(x), address(h), address(qkv),
        address(heads), address(act), address(scaled_a), address(scaled_b), tuning.stream_target_ctas(dev),
        gemm.STREAM_MAX_ROWS, tuning.STREAM_LATE_TRIGGER_BYTES, mma, tcgen05,
        attn_ops._device_error_address(dev), L.stream_handle().value or 0)
    launches = ctypes.c_long(0)
    rc = L.core().dsp_dense_layers(step, (ctypes.c_char * len(table)).from_buffer(table), ctypes.byref(launches))
    L.check(rc, launches=launches.value)
    return True
