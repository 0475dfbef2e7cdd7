"""The few-row product beyond 128 rows: tiles of 192 columns, chunks of rows, K split over clusters and not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("M,N,K,bias,resid,swiglu", [
    (129, 2048, 1536, True, False, False),   # one chunk of 192 columns, the last mostly empty, K split
    (192, 1536, 8960, False, True, False),   # a whole chunk, K split with a residual
    (193, 1536, 1536, True, True, False),    # two chunks of 97
    (385, 256, 4096, False, True, False),    # three chunks of 129
    (536, 4608, 256, True, False, False),    # more tiles than SMs: no split
    (450, 20000, 136, True, True, False),    # several tiles a CTA, a residual, a ragged K
    (300, 1000, 200, True, True, False),     # a last block of W that is not full
    (200, 501, 72, True, True, False),       # single outputs a thread (rows that are no whole pieces)
    (160, 17920, 96, False, False, True),
    (400, 4096, 512, False, False, True),
])
def test_more_rows_than_a_tile(M, N, K, bias, resid, swiglu):
    from dispec_b200.ops import gemm, library
    x, w = rnd((M, K), 1), rnd((N, K), 2, K ** -0.5)
    x[M - 1] *= 3.0
    b, r = rnd((N,), 3) if bias else None, rnd((M, N), 4) if resid else None
    out = torch.full((M, N // 2 if swiglu else N), float("nan"), dtype=torch.bfloat16, device=DEV)
    gemm._stream(x, w, b, r, out, epilogue=gemm.EPI_SWIGLU if swiglu else gemm.EPI_PLAIN)
    assert library.device_error() == 0
    ref = x.double() @ w.double().T
    if swiglu:
        v = ref.view(M, N // 32, 2, 16)
        ref = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(M, -1)
    if bias:
        ref += b.double()
    if resid:
        ref += r.double()
    # the 32-bit sums are within K 2^-24 of sums of magnitude 1; the rounding to bfloat16 is 2^-9 of the result
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all()
    out32 = torch.full((M, N), float("nan"), dtype=torch.float32, device=DEV)
    if not swiglu:
        gemm._stream(x, w, b, None, out32)
        ref32 = x.double() @ w.double().T + (b.double() if bias else 0.0)
        assert ((out32.double() - ref32).abs() <= 1e-4 * (1.0 + ref32.abs())).all()
    # a row does not depend on where it stands among the others of its chunk
    again = torch.empty_like(out)
    gemm._stream(x.flip(0).contiguous(), w, b, r.flip(0).contiguous() if resid else None, again,
                 epilogue=gemm.EPI_SWIGLU if swiglu else gemm.EPI_PLAIN)
    assert torch.equal(again.flip(0), out)


@pytest.mark.parametrize("M,N,K,few", [(137, 1536, 8960, True), (137, 17920, 1536, False), (536, 1536, 8960, True),
                                       (536, 2048, 1536, False), (2048, 1536, 8960, False), (4500, 1536, 1536, False),
                                       # where the other kernel was measured a tenth slower or more
                                       (384, 2048, 1536, False), (384, 1536, 1536, True), (900, 512, 4096, True),
                                       (300, 3584, 18944, True), (385, 3584, 18944, False), (1152, 1536, 8960, True),
                                       (1500, 1536, 8960, False), (384, 4608, 3584, True), (450, 4096, 4096, False)])
def test_which_kernel_runs(M, N, K, few):
    from dispec_b200.ops import tuning
    assert tuning.rows_in_chunks_is_faster(M, N, K, torch.device(DEV)) is few
