"""The product on CTA pairs: chunks of rows, splits of K, blocks of W that are not full, ragged K, every epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("M,N,K,bias,resid,act,dtype", [
    (32, 256, 64, False, False, "", torch.bfloat16),      # one tile of 32 columns, half a ring slot
    (129, 260, 136, True, True, "", torch.bfloat16),      # a second block of W with four rows, ragged K
    (256, 384, 192, True, False, "", torch.float32),      # a whole chunk, the second block's upper half empty
    (257, 512, 1536, False, True, "", torch.float32),     # two chunks of 129, K split
    (300, 9000, 72, True, True, "", torch.bfloat16),      # several tiles a pair
    (513, 640, 2048, False, True, "", torch.bfloat16),
    (200, 512, 1024, False, False, "silu", torch.bfloat16),
    (410, 20480, 128, False, False, "gelu_tanh", torch.bfloat16),
])
@pytest.mark.parametrize("splits", [0, 1, 2, 3, 4])
def test_against_64_bits(M, N, K, bias, resid, act, dtype, splits):
    from dispec_b200.ops import gemm, library
    if splits > 1 and (-(-K // 128) < 2 * splits or N > 2000):
        pytest.skip("too few blocks of k, or more tiles than clusters")
    x, w = rnd((M, K), 1), rnd((N, K), 2, K ** -0.5)
    x[M - 1] *= 3.0
    b, r = rnd((N,), 3) if bias else None, rnd((M, N), 4).to(dtype) if resid else None
    out = torch.full((M, N // 2 if act else N), float("nan"), dtype=dtype, device=DEV)
    epilogue = {"": gemm.EPI_PLAIN, "silu": gemm.EPI_SWIGLU, "gelu_tanh": gemm.EPI_GEGLU}[act]
    gemm._pairs(x, w, b, r, out, epilogue=epilogue, splits=splits)
    assert library.device_error() == 0
    ref = x.double() @ w.double().T
    if act:
        v = ref.view(M, N // 32, 2, 16)
        f = torch.nn.functional.silu if act == "silu" else (lambda t: torch.nn.functional.gelu(t, approximate="tanh"))
        ref = (f(v[:, :, 0]) * v[:, :, 1]).reshape(M, -1)
    if bias:
        ref += b.double()
    if resid:
        ref += r.double()
    # sums of magnitude 1 (3 in the last row) within K 2^-24, the rounding to bfloat16 2^-9 of the result
    tol = 1e-4 * (1.0 + ref.abs()) if dtype == torch.float32 else 2.0 ** -8 * ref.abs() + 1e-3
    assert ((out.double() - ref).abs() <= tol).all()


def test_the_choice_and_what_it_refuses():
    from dispec_b200.ops import gemm, library, tuning
    assert tuning.pairs_are_faster(768, 1536, 1536) and tuning.pairs_are_faster(450, 3584, 18944)
    assert not tuning.pairs_are_faster(4500, 17920, 1536) and not tuning.pairs_are_faster(2048, 2048, 1536)
    x, w = rnd((300, 1536), 5), rnd((1536, 1536), 6, 0.02)
    wide = torch.zeros((300, 1539), dtype=torch.bfloat16, device=DEV)
    for out in (wide[:, 1:1537], wide[:, :1536]):  # columns, or rows, that do not begin on eight bytes: another kernel
        assert not gemm.pairs_supported(x, w, None, None, out)
        with pytest.raises(library.KernelError, match="rows of four outputs"):
            gemm._pairs(x, w, None, None, out)
        assert torch.allclose(gemm.linear(x, w, out=out).float(), (x.double() @ w.double().T).float(), atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("M,N,K", [(129, 260, 136), (300, 1024, 1024), (1024, 512, 64), (1025, 512, 64)])
def test_xielu_in_the_epilogue_and_behind_the_product(M, N, K):
    from dispec_b200.ops import gemm, library, norm32
    x, w, params = rnd((M, K), 7, 3.0), rnd((N, K), 8, K ** -0.5), torch.tensor([0.3, -0.7], device=DEV)
    out = gemm.linear_xielu(x, w, params)
    assert library.device_error() == 0
    z = x.double() @ w.double().T
    p, q = torch.nn.functional.softplus(params.double())
    ref = torch.where(z > 0, p * z * z, (0.5 + q) * (torch.expm1(z.clamp(max=0)) - z)) + z / 2
    # the sums within 1e-5, a slope of at most 2 p |z| + 1/2 + q, one rounding to bfloat16
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * (2 * p * z.abs() + 1.5)).all()
    if M <= 1024:
        sums = gemm._pairs(x, w, None, None, torch.empty((M, N), device=DEV))
        assert torch.equal(out, norm32.xielu(sums, params, torch.bfloat16))
