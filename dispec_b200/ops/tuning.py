"""Launch-shape choices of the kernels, in one place, keyed by quantities of the launch (bytes,
rows, resident CTA slots, keys per CTA) and by the device's SM count, never by a model.

Every constant says what was measured.  None of them bears on correctness: the kernels take any
value that passes their own argument checks and give the same result bit for bit, except where
a split count changes the order of a 32-bit sum.
"""
from __future__ import annotations

import functools

import torch

_sm_count: dict[int, int] = {}


def sm_count(device=None) -> int:
    """Streaming multiprocessors of the device (asked once per device)."""
    index = device.index if isinstance(device, torch.device) else None if device is None else torch.device(device).index
    if index is None:
        index = torch.cuda.current_device()
    if index not in _sm_count:
        _sm_count[index] = int(torch.cuda.get_device_properties(index).multi_processor_count)
    return _sm_count[index]


# ---- few-row matrix product (gemm_stream.cu) ------------------------------------------------
# Its CTAs keep about 100 KB of W on their way each, so two are resident per SM (the second slot is
# for the next kernel's CTAs, which fill their rings while this kernel drains).  K is split over a
# cluster until the launch has one CTA per SM; measured at 8 and at 64 rows: splitting further, to
# both resident slots, is slower (the gate/up product of 140 blocks cut in two: 8 % on the whole step).
STREAM_CTAS_PER_SM = 1


def stream_target_ctas(device=None) -> int:
    return STREAM_CTAS_PER_SM * sm_count(device)


# A product that streams at least this many bytes of W lets its successor start (programmatic
# dependent launch) only once its last tile of W is requested: what the successor requests before
# its own wait would otherwise compete with a long stream.  Shorter products let it start at once.
# Measured on captured decode steps, 8 rows: products of 4.7 to 6.3 MB are faster with the early
# trigger, products of 27 MB and more with the late one (1.334 -> 1.312 ms a step at 28 layers).
STREAM_LATE_TRIGGER_BYTES = 16 << 20

def rows_in_chunks_is_faster(M: int, N: int, K: int, device=None, chunk_rows: int = 128) -> bool:
    """Whether the few-row product beats the many-row product at M rows (always up to ``chunk_rows``); the
    estimate stands beside the kernel (``dsp_gemm_few_rows_faster`` in csrc/gemm_stream.cu)."""
    return M <= chunk_rows or _few_rows_faster(M, N, K, sm_count(device))


@functools.lru_cache(maxsize=4096)
def _few_rows_faster(M: int, N: int, K: int, sms: int) -> bool:
    from dispec_b200.ops import library
    answer = library.core().dsp_gemm_few_rows_faster(M, N, K, STREAM_CTAS_PER_SM * sms)
    if answer < 0:  # (an exception is not kept by the cache)
        library.check(answer, launches=0)
    return bool(answer)


BF16_RESULT, FLOAT32_RESULT, GATED_RESULT, XIELU_RESULT = 0, 1, 2, 3  # what the time of a product is fitted for


def pairs_are_faster(M: int, N: int, K: int, device=None, result: int = BF16_RESULT) -> bool:
    """Whether the product on CTA pairs with swapped roles beats the one that runs otherwise at M rows; the
    estimate stands beside the kernel (``dsp_gemm_pairs_faster`` in csrc/gemm_pairs.cu)."""
    return _pairs_faster(M, N, K, sm_count(device), result)


@functools.lru_cache(maxsize=4096)
def _pairs_faster(M: int, N: int, K: int, sms: int, result: int) -> bool:
    from dispec_b200.ops import library
    answer = library.core().dsp_gemm_pairs_faster(M, N, K, STREAM_CTAS_PER_SM * sms, result)
    if answer < 0:  # (an exception is not kept by the cache)
        library.check(answer, launches=0)
    return bool(answer)


def many_rows_product(M: int, N: int, K: int, result: int, device) -> str:
    """The kernel of a bfloat16 product of more rows than the few-row kernel always takes: "pairs", "stream" or "tcgen05"
    (a product of a step asks once, for its size and kind of result)."""
    return _many_rows_product(M, N, K, result, sm_count(device))


@functools.lru_cache(maxsize=4096)
def _many_rows_product(M: int, N: int, K: int, result: int, sms: int) -> str:
    if _pairs_faster(M, N, K, sms, result):
        return "pairs"
    return "stream" if result != GATED_RESULT and _few_rows_faster(M, N, K, sms) else "tcgen05"


# ---- attention of single tokens (attn_mma.cu, decode kernel) ---------------------------------
ATTN_CTAS_PER_SM = 2  # resident CTAs the decode launch aims for
CLUSTER_MAX_SPLITS = 8  # key splits of one row that merge on chip (one thread-block cluster)
SPLIT_MIN_KEYS = 256  # a split is not worth less than this many keys
MAX_OUTER = 32  # key ranges per row beyond the cluster
OUTER_MIN_KEYS = 256  # a CTA of a row cut into ranges still reads at least this many keys
MAX_SPLITS = 32  # splits merged from global scratch (groups too large for the cluster kernels)


def attention_target_ctas(device=None) -> int:
    return ATTN_CTAS_PER_SM * sm_count(device)


def choose_splits(num_rows: int, num_kv_heads: int, max_ctx: int, target_ctas: int,
                  limit: int = CLUSTER_MAX_SPLITS) -> int:
    """Key splits for single-token rows so that rows x KV heads x splits covers ``target_ctas``
    (``attention_target_ctas(device)``) once, each split keeping at least ``SPLIT_MIN_KEYS`` keys.  Measured at 1,100 keys and
    128-wide heads, 2 KV heads: the best count keeps the launch within two CTAs per SM (8 splits
    at 8 rows, 4 at 32, 2 at 64, 1 at 128)."""
    if num_rows <= 0:
        return 1
    want = max(1, target_ctas // (num_rows * num_kv_heads))
    return max(1, min(want, limit, -(-max_ctx // SPLIT_MIN_KEYS)))


def choose_outer(num_rows: int, num_kv_heads: int, max_ctx: int, splits: int, target_ctas: int) -> int:
    """Key ranges per single-token row on top of the cluster's ``splits``: when a full cluster
    per row and KV head still leaves SMs idle (few rows) and the context is long enough to share.
    Measured at 128-wide heads: the best count brings the launch to about two CTAs per SM (16
    ranges for one row of 32,768 keys, 2 for 8 rows), as long as a CTA keeps ``OUTER_MIN_KEYS``."""
    if num_rows <= 0 or splits < CLUSTER_MAX_SPLITS:
        return 1
    want = target_ctas // (num_rows * num_kv_heads * splits)
    return max(1, min(want, MAX_OUTER, max_ctx // (splits * OUTER_MIN_KEYS)))
