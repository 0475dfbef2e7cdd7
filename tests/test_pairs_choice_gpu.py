"""Where the product on CTA pairs is chosen, and how far 32-bit results lie from 64 bits then."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K,result,pairs", [
    (1032, 4096, 1024, 0, False), (1032, 4096, 1024, 2, False), (897, 6144, 1536, 2, False),  # 1.1 to 1.3 times as long
    (137, 5120, 13824, 2, True),  # a gated product has no few-row kernel to stay with
    (225, 4608, 3584, 1, False), (289, 4608, 3584, 1, False),
    (536, 1536, 1536, 0, True), (536, 1536, 1536, 1, True), (2100, 1536, 1536, 0, False),
])
def test_the_choice(M, N, K, result, pairs):
    from dispec_b200.ops import tuning
    assert tuning.pairs_are_faster(M, N, K, result=result) == pairs
    assert (tuning.many_rows_product(M, N, K, result, torch.device(DEV)) == "pairs") == pairs


@pytest.mark.parametrize("M,N,K,fused", [(137, 8960, 1536, True), (900, 4096, 1024, False), (900, 14336, 4096, True),
                                         (2048, 14336, 4096, True), (2500, 8960, 1536, False), (128, 8960, 1536, False)])
def test_xielu_is_fused_where_that_is_faster(M, N, K, fused, monkeypatch):
    from dispec_b200.ops import gemm
    x, w = (torch.ones(s, dtype=torch.bfloat16, device=DEV) for s in ((M, K), (N, K)))
    asked, pairs = [], gemm._pairs
    monkeypatch.setattr(gemm, "_pairs", lambda *a, **k: asked.append(k.get("epilogue", 0)) or pairs(*a, **k))
    gemm.linear_xielu(x, w, torch.tensor([0.3, -0.7], device=DEV))
    assert (gemm.EPI_XIELU in asked) == fused


@pytest.mark.parametrize("M,N,K", [(225, 4608, 3584), (300, 1536, 8960), (193, 1024, 4096), (1153, 512, 2048), (640, 1536, 1536)])
def test_32_bit_results_lose_nothing(M, N, K):
    """The tensor cores cut every sum off: a kernel that adds more of K one after the other is not chosen for its speed."""
    from dispec_b200.ops import gemm, tuning
    g = torch.Generator(device=DEV).manual_seed(N + K)
    x, w = (torch.rand(s, generator=g, device=DEV).to(torch.bfloat16) for s in ((M, K), (N, K)))
    ref = x.double() @ w.double().T
    other = gemm._stream if tuning.rows_in_chunks_is_faster(M, N, K, torch.device(DEV)) else gemm._tcgen05
    error = lambda out: float(((out.double() - ref) / ref).abs().mean())
    mine = error(gemm.linear(x, w, out_dtype=torch.float32))
    assert mine <= 1.05 * error(other(x, w, None, None, torch.empty((M, N), device=DEV)))
