"""y = x W^T (+ bias) (+ residual): the one matrix product the model uses.

float32: every operand cut into three bfloat16 pieces that add up to it, whose products run on the
tensor cores and are summed in 32 bits (``dsp_gemm_split``: closer to 64 bits than a chain of 32-bit
FMAs); the FMA kernel (``dsp_gemm_simt``) for K below 1,536 and for matrices that TMA cannot read.  Which of
the two runs is decided by the matrix alone, and a row does not depend on its batch in either.
bfloat16: the weight-streaming tcgen05 kernel for up to 128 rows (decoding and the rows whose
logits are wanted); above that the persistent tcgen05/TMA kernel of this package, except that, mostly
at some hundred rows, the kernel on CTA pairs with swapped roles (it splits K, and cuts the rows into
equal chunks) or the weight-streaming kernel runs where ``tuning.many_rows_product`` says so.  Operands
those kernels cannot take (a width that is no multiple of 8) go to the FMA kernel when there
are at most 64 rows or 32-bit logits are wanted, and otherwise to the library matrix product
(cuBLAS through torch.mm), which is where the reference engine itself calls a library
(puneethgv/DiSpec dispec/engine/model_runner.py:132,158,225-226,231).  ``backend=`` names a kernel outright (tests and
comparisons).
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass

import torch

from dispec_b200.ops import library as L
from dispec_b200.ops import tuning

STREAM_MAX_ROWS = 128  # rows up to which the weight-streaming kernel always runs
SPLIT_MIN_K = 1536  # length of a product of floats from which the tensor cores are used
NORM_SPLIT_MAX_ROWS = 64  # rows up to which a norm is split over two products


@dataclass
class NormedRows:
    """The input of a product, given as a norm that is still to be applied:
    weight * (source * rsqrt(mean(source^2) + eps)).  ``scaled`` = round(source) * weight in the
    storage type, if the product that wrote ``source`` stored it as well: then a few-row product
    multiplies ``scaled`` by its matrix and its result rows by the rsqrt factors (which it forms
    itself from ``source`` while the matrix streams), and the norm needs no kernel of its own.
    Every other consumer calls ``materialize()``, which runs the norm kernel."""
    source: torch.Tensor
    weight: torch.Tensor
    eps: float
    scaled: torch.Tensor | None = None

    @property
    def shape(self):
        return self.source.shape

    @property
    def dtype(self):
        return self.source.dtype

    @property
    def device(self):
        return self.source.device

    def materialize(self) -> torch.Tensor:
        from dispec_b200.ops.elementwise import rms_norm
        return rms_norm(self.source, self.weight, self.eps)

    def splittable(self, w: torch.Tensor) -> bool:
        """Whether the few-row kernel can take this norm apart (see the class text)."""
        x = self.scaled
        M, K = self.source.shape
        return (x is not None and x.dtype == torch.bfloat16 and M <= NORM_SPLIT_MAX_ROWS
                and self.source.stride(1) == 1 and self.source.stride(0) % 8 == 0
                and self.source.data_ptr() % 16 == 0 and stream_supported(M, K, x, w))
EPI_PLAIN, EPI_SWIGLU, EPI_GEGLU, EPI_XIELU = 0, 1, 2, 3
SWIGLU_BLOCK = 16  # gate/up rows alternate in blocks of this many for the fused epilogue


def _simt(x, w, bias, residual, out, tile: int = -1):
    """``tile``: a tile of the kernel by index instead of its own choice (comparisons; the same bits)."""
    M, K = x.shape
    N = w.shape[0]
    L.check(L.core().dsp_gemm_simt(
        L.ptr(x), L.i64(x.stride(0)), L.ptr(w), L.ptr(bias), L.ptr(residual),
        L.i64(residual.stride(0) if residual is not None else 0), L.ptr(out), L.i64(out.stride(0)),
        M, N, K, L.dtype_code(x.dtype), L.dtype_code(out.dtype), tile, L.stream_handle()))
    return out


def _split(x, w, bias, residual, out):
    """The product of floats on the tensor cores, operands cut into three bfloat16 pieces."""
    M, K = x.shape
    L.check(L.core().dsp_gemm_split(
        L.ptr(x), L.i64(x.stride(0)), L.ptr(w), L.ptr(bias), L.ptr(residual),
        L.i64(residual.stride(0) if residual is not None else 0), L.ptr(out), L.i64(out.stride(0)),
        M, w.shape[0], K, L.stream_handle()))
    return out


def _pairs(x, w, bias, residual, out, epilogue=EPI_PLAIN, splits: int = 0, chunks: int = 0, act: torch.Tensor | None = None):
    """The product of some hundred rows on CTA pairs; ``act``: the raw parameters of ``EPI_XIELU``; ``splits``, ``chunks``: instead of its own choice (comparisons)."""
    M, K = x.shape
    L.check(L.core().dsp_gemm_pairs(
        L.ptr(x), L.i64(x.stride(0)), L.ptr(w), L.ptr(bias), L.ptr(residual),
        L.i64(residual.stride(0) if residual is not None else 0), L.ptr(out), L.i64(out.stride(0)),
        M, w.shape[0], K, L.dtype_code(out.dtype), epilogue, L.ptr(act), splits, chunks, L.stream_handle()))
    return out


def _tcgen05(x, w, bias, residual, out, pairs: bool = True, epilogue=EPI_PLAIN):
    """The many-row product; ``pairs``: CTA pairs (cta_group::2), the default, or single CTAs."""
    M, K = x.shape
    N = w.shape[0]
    L.check(L.core().dsp_gemm_tcgen05(
        L.ptr(x), L.i64(x.stride(0)), L.ptr(w), L.ptr(bias), L.ptr(residual),
        L.i64(residual.stride(0) if residual is not None else 0), L.ptr(out), L.i64(out.stride(0)),
        M, N, K, L.dtype_code(out.dtype), int(pairs), epilogue, L.stream_handle()))
    return out


def _stream(x, w, bias, residual, out, epilogue=EPI_PLAIN, target_ctas: int | None = None,
            norm: NormedRows | None = None, scaled_out: tuple | None = None):
    """The few-row product; ``target_ctas``: resident CTA slots the launch may fill by splitting K
    over a cluster (default: one per SM of the device).  ``norm``: x is ``norm.scaled`` and the
    result rows take the norm's rsqrt factors.  ``scaled_out`` = (gain, out2): out2 = out * gain."""
    M = x.shape[0]
    N, K = w.shape
    if target_ctas is None:
        target_ctas = tuning.stream_target_ctas(x.device)
    src = norm.source if norm is not None else None
    gain2, out2 = scaled_out if scaled_out is not None else (None, None)
    L.check(L.core().dsp_gemm_stream(
        L.ptr(x), L.i64(x.stride(0)), L.ptr(w), L.ptr(bias), L.ptr(residual),
        L.i64(residual.stride(0) if residual is not None else 0), L.ptr(out), L.i64(out.stride(0)),
        M, N, K, L.dtype_code(out.dtype), target_ctas, epilogue,
        L.i64(tuning.STREAM_LATE_TRIGGER_BYTES), L.ptr(src), L.i64(src.stride(0) if src is not None else 0),
        ctypes.c_float(norm.eps if norm is not None else 0.0), L.ptr(gain2), L.ptr(out2),
        L.i64(out2.stride(0) if out2 is not None else 0), L.stream_handle()))
    return out


def split_supported(w: torch.Tensor) -> bool:
    """Whether a product of floats runs on the tensor cores: by its matrix alone, so that a row has the same bits
    alone and among others.  Below ``SPLIT_MIN_K`` a few rows wait longer for that kernel's fixed latencies than for the
    FMA chain: 4 rows x 1,536 x 512 8.0 us for 4.4, x 1,024 9.5 for 7.9, x 1,280 10.3 for 9.6, x 1,536 11.4 for 11.3 (264 rows
    14 and 18, 15 and 33, 17 and 41, 18 and 49); nor is it always closer to 64 bits there (products of two lognormal
    operands of sigma 2, K 256 / 512 / 1,024: 7.5e-7 / 7.1e-7 / 9.1e-7 off for 3.4e-7 / 3.7e-7 / 6.8e-7 of the chain; from
    1,280 on it is, with eight distributions tried)."""
    return w.shape[1] >= SPLIT_MIN_K and w.shape[1] % 4 == 0 and w.data_ptr() % 16 == 0


def tcgen05_supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    return (x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and x.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def pairs_supported(x: torch.Tensor, w: torch.Tensor, bias, residual, out: torch.Tensor) -> bool:
    """Whether the operands of a product let the kernel on CTA pairs finish four outputs of a row at a time."""
    return tcgen05_supported(x, w) and _whole_fours(w, bias, residual, out)


def _whole_fours(w: torch.Tensor, bias, residual, out: torch.Tensor) -> bool:
    width = 4 * out.element_size()
    return (w.shape[0] % 4 == 0 and out.stride(0) % 4 == 0 and out.data_ptr() % width == 0
            and (residual is None or (residual.stride(0) % 4 == 0 and residual.data_ptr() % width == 0))
            and (bias is None or bias.data_ptr() % 8 == 0))


def stream_supported(M: int, K: int, x: torch.Tensor, w: torch.Tensor) -> bool:
    return (M <= STREAM_MAX_ROWS and K % 8 == 0 and x.stride(0) % 8 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def gate_up_swiglu_supported(x, w: torch.Tensor) -> bool:
    """Whether act(gate) * up can be formed in the epilogue of the gate/up product."""
    M, K = x.shape
    if x.dtype != torch.bfloat16 or w.shape[0] % 32:
        return False
    if isinstance(x, NormedRows):
        x = x.scaled if x.splittable(w) else x.source
    if M <= STREAM_MAX_ROWS:
        return stream_supported(M, K, x, w)
    return tcgen05_supported(x, w)


def linear_gate_up_swiglu(x, w_interleaved, out=None, act: str = "silu"):
    """act(x Wg^T) * (x Wu^T) in one kernel (``act`` "silu" or "gelu_tanh"): ``w_interleaved`` holds 16 gate rows, the 16 up
    rows of the same outputs, the next 16 gate rows, ...  Returns [M, N/2].  ``x``: a tensor or
    ``NormedRows``."""
    assert gate_up_swiglu_supported(x, w_interleaved)
    norm = None
    if isinstance(x, NormedRows):
        if x.splittable(w_interleaved):
            norm, x = x, x.scaled
        else:
            x = x.materialize()
    M, N = x.shape[0], w_interleaved.shape[0]
    if out is None:
        out = torch.empty((M, N // 2), dtype=x.dtype, device=x.device)
    epilogue = {"silu": EPI_SWIGLU, "gelu_tanh": EPI_GEGLU}[act]
    if M > STREAM_MAX_ROWS:
        if (tuning.many_rows_product(M, N, x.shape[1], tuning.GATED_RESULT, x.device) == "pairs"
                and _whole_fours(w_interleaved, None, None, out)):
            return _pairs(x, w_interleaved, None, None, out, epilogue=epilogue)
        return _tcgen05(x, w_interleaved, None, None, out, epilogue=epilogue)
    return _stream(x, w_interleaved, None, None, out, epilogue=epilogue, norm=norm)


def linear_xielu(x: torch.Tensor, w: torch.Tensor, params: torch.Tensor) -> torch.Tensor:
    """xIELU(x W^T), the activation formed in 32 bits from the 32-bit sums and rounded to x's type (``params``: its two raw
    parameters, float32): in the epilogue of the product on CTA pairs, or by a kernel of its own behind a product with a
    32-bit result, whichever the estimate beside the former says is faster (``tuning.XIELU_RESULT``).  The activation is
    the same function of the sums in both; the sums are added in the order of the kernel that runs.  us, fused and not, w
    8,960 x 1,536: 137 rows 16 and 17, 300 21 and 22, 536 34 and 31, 1,016 46 and 49; w 14,336 x 4,096: 536 rows 68 and 82,
    2,048 171 and 216; w 4,096 x 1,024: 900 rows 30 and 24."""
    from dispec_b200.ops.norm32 import xielu
    if not (x.is_cuda and w.is_cuda and params.is_cuda):
        raise L.KernelError("linear_xielu: CUDA tensors only (there is no CPU path)")
    assert x.dim() == 2 and w.dim() == 2 and x.shape[1] == w.shape[1], (x.shape, w.shape)
    assert x.stride(1) == 1 and w.is_contiguous() and x.dtype == w.dtype
    M, N = x.shape[0], w.shape[0]
    if (M > STREAM_MAX_ROWS and x.dtype == torch.bfloat16 and tcgen05_supported(x, w)
            and tuning.pairs_are_faster(M, N, x.shape[1], x.device, tuning.XIELU_RESULT)):
        out = torch.empty((M, N), dtype=x.dtype, device=x.device)
        if _whole_fours(w, None, None, out):
            assert params.dtype == torch.float32 and params.numel() == 2 and params.is_contiguous()
            return _pairs(x, w, None, None, out, epilogue=EPI_XIELU, act=params)
    return xielu(linear(x, w, out_dtype=torch.float32), params, x.dtype)


def _library(x, w, bias, residual, out):
    """The library matrix product; bias and residual are folded in by the library as well."""
    assert out.dtype == torch.bfloat16
    if residual is not None:
        if out.data_ptr() != residual.data_ptr():
            out.copy_(residual)
        out.addmm_(x, w.t())
        if bias is not None:
            out.add_(bias)
    elif bias is not None:
        torch.addmm(bias, x, w.t(), out=out)
    else:
        torch.mm(x, w.t(), out=out)
    return out


def linear(x, w: torch.Tensor, bias: torch.Tensor | None = None,
           residual: torch.Tensor | None = None, out_dtype: torch.dtype | None = None,
           out: torch.Tensor | None = None, backend: str | None = None, then_norm=None):
    """x [M, K] (row stride free, unit column stride), w [N, K] contiguous, bias [N],
    residual [M, N] of the output type.  Output type: ``out_dtype`` (default: x's);
    bfloat16 inputs may produce float32 (logits).  ``backend``: "stream", "tcgen05", "pairs",
    "library" or "simt" instead of the choice described at the top of this file.

    ``x`` may be ``NormedRows`` (a norm still to be applied): the few-row kernel takes it apart
    where it can, otherwise the norm kernel runs first.  ``then_norm`` = (weight, eps) of the
    norm that follows this product: the call returns (out, NormedRows of out), with the scaled
    copy filled in where the few-row kernel wrote it."""
    norm = None
    if isinstance(x, NormedRows):
        if backend in (None, "stream") and x.splittable(w):
            norm, x, backend = x, x.scaled, "stream"
        else:
            x = x.materialize()
    if not (x.is_cuda and w.is_cuda):
        raise L.KernelError("linear: CUDA tensors only (there is no CPU path)")
    assert x.dim() == 2 and w.dim() == 2 and x.shape[1] == w.shape[1], (x.shape, w.shape)
    assert x.stride(1) == 1 and w.is_contiguous() and x.dtype == w.dtype
    M, K = x.shape
    N = w.shape[0]
    out_dtype = out_dtype or (out.dtype if out is not None else x.dtype)
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=x.device)
    assert out.shape == (M, N) and out.stride(1) == 1 and out.dtype == out_dtype
    if bias is not None:
        assert bias.shape == (N,) and bias.dtype == x.dtype and bias.is_contiguous()
    if residual is not None:
        assert residual.shape == (M, N) and residual.dtype == out_dtype and residual.stride(1) == 1

    def result(scaled=None):
        if then_norm is None:
            return out
        return out, NormedRows(out, then_norm[0], then_norm[1], scaled)

    if M == 0:
        return result()
    if x.dtype == torch.float32:
        assert out_dtype == torch.float32
        (_split if split_supported(w) and backend != "simt" else _simt)(x, w, bias, residual, out)
        return result()
    if backend is None:
        if stream_supported(M, K, x, w):
            backend = "stream"
        elif M > STREAM_MAX_ROWS and tcgen05_supported(x, w):  # ("stream": a norm after it runs as a kernel)
            result_kind = tuning.FLOAT32_RESULT if out_dtype == torch.float32 else tuning.BF16_RESULT
            backend = tuning.many_rows_product(M, N, K, result_kind, x.device)
            if backend == "pairs" and not _whole_fours(w, bias, residual, out):
                backend = "stream" if tuning.rows_in_chunks_is_faster(M, N, K, x.device, STREAM_MAX_ROWS) else "tcgen05"
        elif M > STREAM_MAX_ROWS and out_dtype == torch.bfloat16:
            backend = "library"
        else:
            backend = "simt"
    if backend == "stream":
        scaled = None
        if (then_norm is not None and M <= NORM_SPLIT_MAX_ROWS and out_dtype == torch.bfloat16
                and then_norm[0].dtype == torch.bfloat16):
            scaled = torch.empty((M, N), dtype=out_dtype, device=x.device)
        _stream(x, w, bias, residual, out, norm=norm,
                scaled_out=(then_norm[0], scaled) if scaled is not None else None)
        return result(scaled)
    if backend == "tcgen05":
        _tcgen05(x, w, bias, residual, out)
    elif backend == "pairs":
        _pairs(x, w, bias, residual, out)
    elif backend == "library":
        _library(x, w, bias, residual, out)
    elif backend == "simt":
        _simt(x, w, bias, residual, out)
    else:
        raise ValueError(f"unknown backend {backend!r}")
    return result()
