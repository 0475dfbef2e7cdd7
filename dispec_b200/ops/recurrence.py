"""Linear attention as a recurrence over a per-request matrix state (32-bit, FMA units):
S_t = diag(a_t) S_(t-1) + b_t v_t^T,  o_t = S_t^T q_t  (``csrc/linear_recurrence.cu``), and the gated delta
rule, whose write depends on what the state already holds (``csrc/delta_rule.cu``)."""
from __future__ import annotations

import ctypes

import torch

from dispec_b200.ops import library as L

FIXED_DECAY, FORGET_GATE, KEY_DECAY, STEP_DECAY = 0, 1, 2, 3
# A request of SEGMENTS_MIN_TOKENS and more in a step is cut into segments that run side by side, where its heads alone leave
# SMs idle: a request's tokens one after the other take 102 (one decay a head) or 127 ns each, whoever shares the step, the
# segments' products some 80 together.  us in segments and in one piece, 12 heads of 128 x 128, fixed decay / forget gate: 512
# tokens 56 and 58 / 59 and 69, 768 66 and 83 / 70 and 100, 2,048 162 and 213 / 180 and 263; 833 and 1,667 tokens 198 and 277 /
# 218 and 335; 24 heads of 64 x 64, 1,024 tokens 71 and 112; 4 heads, 33 and 106.  Several requests of one length fill the SMs
# by themselves: three of 768 182 and 140 / 196 and 174, eight of 1,024 601 and 541 / 660 and 657.  The rule looks at the request
# alone nevertheless, so that its bits do not depend on who shares the step.  More blocks, or more state rows, lose: 64 heads
# of 128 x 64, 1,024 tokens 261 and 211; 6 heads of 256 x 256, twice 768 204 and 189.
SEGMENTS_MIN_TOKENS = 768  # a multiple of 64, the length of a segment
_MAX_SEGMENTS = 128  # of a request: longer segments rather than more of them, since a state is kept for each
_SEGMENTS_MAX_ROWS = 128  # state rows
_SEGMENTS_MAX_BLOCKS = 96  # blocks of 16 value columns, over all heads
_SEGMENTS_BYTES = 256 << 20  # workspace; with more, groups of heads follow one another


def _segment_floats(T: int, heads: int, dim: int, vdim: int) -> int:
    """Workspace for the segments of ``heads`` heads of a step of T tokens."""
    question = L.mixer_library("linear_recurrence").dsp_linear_recurrence_segment_floats
    question.restype = ctypes.c_long
    return question(T, heads, dim, vdim, SEGMENTS_MIN_TOKENS)


def _cut_into_segments(num_heads: int, dim: int, vdim: int) -> bool:
    return dim <= _SEGMENTS_MAX_ROWS and num_heads * -(-vdim // 16) <= _SEGMENTS_MAX_BLOCKS


def linear_recurrence(proj: torch.Tensor, q_off: int, k_off: int, v_off: int, mode: int, num_heads: int,
                      dim: int, vdim: int, state: torch.Tensor, state_slot: torch.Tensor,
                      q_start: torch.Tensor, positions: torch.Tensor, *, decay: torch.Tensor | None = None,
                      inv_freq: torch.Tensor | None = None, rot: int = 0, key_scale: float = 1.0,
                      gate_bias: torch.Tensor | None = None, lower: torch.Tensor | None = None,
                      silu_inputs: bool = False, gate_map: torch.Tensor | None = None, low_off: int = 0,
                      q_scale: float = 1.0, power: float = 1.0, steps: torch.Tensor | None = None,
                      skip: torch.Tensor | None = None, num_groups: int = 0,
                      host_q_len: list | None = None) -> torch.Tensor:
    """``proj`` [T, columns]: the raw rows of the mixer's fused projection (query columns from
    ``q_off``, key or forget-gate columns from ``k_off``, value columns from ``v_off``, each head by
    head).  ``state`` float32 [slots, H, dim, vdim] is read and left updated for the sequences of the
    step (``q_start`` [S + 1], ``state_slot`` [S]); a sequence whose first position is negative is
    skipped.  ``host_q_len``: the tokens of each request, where the host knows them (kernels that have nothing to do in this
    step are then not launched).  ``silu_inputs`` (fixed decay only): the raw query, key and value columns pass through
    silu before anything else.  Returns o as float32 [T, H * vdim].

    ``KEY_DECAY``: query columns times ``q_scale``, key columns times ``key_scale``, and a decay per key
    channel sigmoid(z)^power with z = r ``gate_map`` + ``gate_bias``, r the columns of the row from
    ``low_off`` on and ``gate_map`` float32 [rank, H * dim].  ``STEP_DECAY``: ``proj`` float32; query and key
    columns (``dim`` for each of ``num_groups`` groups of heads) are shared by the heads of a group,
    ``steps`` float32 [T, 2, H] holds the factor on the value and the decay of every token and head, and
    ``skip`` float32 [H] times the value is added to o."""
    if not (proj.is_cuda and state.is_cuda):
        raise L.KernelError("linear_recurrence: CUDA tensors only (there is no CPU path)")
    assert proj.dim() == 2 and proj.stride(1) == 1
    assert state.dtype == torch.float32 and state.is_contiguous() and state.shape[1:] == (num_heads, dim, vdim)
    for t in (state_slot, q_start, positions):
        assert t.dtype == torch.int32 and t.is_contiguous()
    for t in (decay, inv_freq, gate_bias, lower, gate_map, steps, skip):
        assert t is None or (t.dtype == torch.float32 and t.is_contiguous() and t.is_cuda)
    S = state_slot.shape[0]
    assert q_start.shape[0] == S + 1
    T = proj.shape[0]
    rank, heads_per_group = 0, 1
    if mode == KEY_DECAY:
        rank = gate_map.shape[0]
        assert gate_map.shape == (rank, num_heads * dim) and gate_bias.shape == (num_heads * dim,)
        assert 0 <= low_off and low_off + rank <= proj.shape[1]
    if mode == STEP_DECAY:
        assert num_groups > 0 and num_heads % num_groups == 0 and proj.dtype == torch.float32
        assert steps.shape == (T, 2, num_heads) and skip.shape == (num_heads,)
        heads_per_group = num_heads // num_groups
    out = torch.empty((T, num_heads * vdim), dtype=torch.float32, device=proj.device)
    lib = L.mixer_library("linear_recurrence")
    # portions of prompts: a first, parallel kernel writes q_t, b_t (a_t) of every token as floats and
    # the sequential kernel streams them; steps of (nearly) single tokens transform while staging
    some_long, all_long = False, False
    if T >= SEGMENTS_MIN_TOKENS and _cut_into_segments(num_heads, dim, vdim):
        longest, shortest = (max(host_q_len), min(host_q_len)) if host_q_len is not None else (T, T if S == 1 else 0)
        some_long, all_long = longest >= SEGMENTS_MIN_TOKENS, shortest >= SEGMENTS_MIN_TOKENS
    scratch = None
    if (T > 2 * S or some_long) and mode != STEP_DECAY:
        planes = 2 if mode == FIXED_DECAY else 3
        scratch = torch.empty((T, planes, num_heads * dim), dtype=torch.float32, device=proj.device)
    segment_scratch, heads = None, 0
    if some_long:
        heads = max(1, min(num_heads, _SEGMENTS_BYTES // (4 * _segment_floats(T, 1, dim, vdim))))
        while segment_scratch is None:
            try:
                segment_scratch = torch.empty(_segment_floats(T, heads, dim, vdim), dtype=torch.float32, device=proj.device)
            except torch.OutOfMemoryError:  # fewer heads at a time give the same bits
                if heads == 1:
                    raise
                heads = (heads + 1) // 2
    L.check(lib.dsp_linear_recurrence(
        L.ptr(proj), L.dtype_code(proj.dtype), L.i64(proj.stride(0)), q_off, k_off, v_off, mode, num_heads, dim,
        vdim, L.ptr(decay), L.ptr(inv_freq), rot, L.f32(key_scale), int(silu_inputs), L.ptr(gate_bias), L.ptr(lower),
        L.ptr(gate_map), low_off, rank, L.f32(q_scale), L.f32(power), L.ptr(steps), L.ptr(skip), heads_per_group, L.ptr(state),
        L.ptr(state_slot), L.ptr(q_start), L.ptr(positions), L.ptr(out), L.i64(out.stride(0)), S, T,
        L.ptr(scratch), L.ptr(segment_scratch), heads, SEGMENTS_MIN_TOKENS, _MAX_SEGMENTS, int(all_long), L.stream_handle()),
        launches=(scratch is not None) + (not all_long) + (3 * -(-num_heads // heads) if some_long else 0))
    return out


DELTA_RUN = 8  # tokens of a portion that the delta rule takes together: the step lists its runs like attention tiles
_DELTA_COEF = 20
_DELTA_MAX_WALK = 256  # state rows up to which portions are taken in runs


def delta_rule(ctx, rows: torch.Tensor, steps: torch.Tensor, num_heads: int, num_groups: int, dim: int, vdim: int,
               state: torch.Tensor) -> torch.Tensor:
    """S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q for every token of the step, in order.

    ``rows`` float32 [T, columns]: q and k (``num_groups`` x ``dim`` each) and v (``num_heads`` x ``vdim``) side by
    side; head h uses q and k of group h // (num_heads / num_groups).  ``steps`` float32 [T, 2, H]: beta and ln g.
    ``state`` float32 [slots, H, dim, vdim] is read and left updated for the step's requests (``ctx``: the
    step's arrays, with its list of runs of ``DELTA_RUN`` tokens); a request whose first position is
    negative is skipped.  Returns o as float32 [T, H * vdim]."""
    if not (rows.is_cuda and state.is_cuda):
        raise L.KernelError("delta_rule: CUDA tensors only (there is no CPU path)")
    H, G, T, S = num_heads, num_groups, rows.shape[0], ctx.state_slot.shape[0]
    assert rows.dtype == torch.float32 and rows.dim() == 2 and rows.stride(1) == 1
    assert rows.shape[1] == 2 * G * dim + H * vdim and H % G == 0
    assert steps.dtype == torch.float32 and steps.shape == (T, 2, H) and steps.is_contiguous()
    assert state.dtype == torch.float32 and state.is_contiguous() and state.shape[1:] == (H, dim, vdim)
    for t in (ctx.state_slot, ctx.q_start, ctx.positions):
        assert t.dtype == torch.int32 and t.is_contiguous()
    out = torch.empty((T, H * vdim), dtype=torch.float32, device=rows.device)
    run_seq, run_tok0, num_runs = ctx.attention_tiles[DELTA_RUN]
    coef = None
    if T > ctx.num_decode_seqs and dim <= _DELTA_MAX_WALK:
        coef = torch.empty((T, H, _DELTA_COEF), dtype=torch.float32, device=rows.device)
    L.check(L.mixer_library("delta_rule").dsp_delta_rule(
        L.ptr(rows), L.i64(rows.stride(0)), 0, G * dim, 2 * G * dim, L.ptr(steps), H, G, dim, vdim, L.ptr(state),
        L.ptr(ctx.state_slot), L.ptr(ctx.q_start), L.ptr(ctx.positions), L.ptr(run_seq), L.ptr(run_tok0), num_runs,
        L.ptr(out), L.i64(out.stride(0)), S, ctx.num_decode_seqs, L.ptr(coef), L.stream_handle()),
        launches=(1 if ctx.num_decode_seqs or coef is None else 0) + (2 if coef is not None else 0))
    return out
