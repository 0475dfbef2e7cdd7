"""The product of floats whose operands are cut into bfloat16 pieces: edges of tiles, chunks of rows and splits of K,
rows alone and among others, operands whose pieces do not hold."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24  # unit roundoff of float32


def rnd(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def run(x, w, b=None, r=None):
    from dispec_b200.ops import gemm, library
    out = gemm._split(x, w, b, r, torch.full((x.shape[0], w.shape[0]), float("nan"), device=DEV))
    assert library.device_error() == 0
    return out


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (16, 128, 32), (17, 129, 36), (32, 127, 128), (33, 260, 132), (64, 640, 516),
                                   (65, 5700, 160),   # no split of K
                                   (96, 1536, 1540),  # K in three splits, a ragged last block
                                   (97, 2048, 512), (193, 300, 1000), (5, 40000, 192)])  # more tiles than SMs
def test_against_64_bits_and_rows_alone(M, N, K):
    x, w, b, r = rnd((M, K), 1), rnd((N, K), 2), rnd((N,), 3), rnd((M, N), 4)
    out = run(x, w, b, r)
    ref = x.double() @ w.double().T + b.double() + r.double()
    # pieces left out: 4 U of a product; each of the 8 sums of 128 k is cut off by at most 2 U; a sum for every 128 k, of
    # the small products, of the splits of K, of bias and residual
    bound = (4 + 16 + K / 128 + 12) * U * (x.abs().double() @ w.abs().double().T + b.abs().double() + r.abs().double())
    assert ((out.double() - ref).abs() <= bound).all()
    for a, n in ((0, 1), (M // 2, 1), (M // 3, 20)):
        part = slice(a, min(M, a + n))
        assert torch.equal(run(x[part].contiguous(), w, b, r[part].contiguous()), out[part])
    odd = torch.zeros((M, K + 1), device=DEV)
    odd[:, 1:] = x  # rows that are no whole 16-byte pieces
    assert torch.equal(run(odd[:, 1:], w, b, r), out)


@pytest.mark.parametrize("M,N", [(3, 300), (40, 9000)])  # K split and not
def test_where_the_pieces_do_not_hold(M, N):
    from dispec_b200.ops import gemm
    K = 512
    x, w = rnd((M, K), 5), rnd((N, K), 6)
    x[0, 5], x[1, 7], x[2, 9] = float("inf"), float("nan"), 3.4e38
    w[3, 1] = float("-inf")
    w[9] *= 2.0 ** 70
    w[12] *= 2.0 ** -80
    out = run(x, w)
    chain = gemm._simt(x, w, None, None, torch.empty_like(out))
    assert torch.equal(out.isnan(), chain.isnan()) and torch.equal(out[chain.isinf()], chain[chain.isinf()])
    assert out[0].isinf().all() or out[0, 3].isnan()
    sized = chain.isfinite() & ((chain.abs() < 2.0 ** -60) | (chain.abs() > 2.0 ** 100))
    assert sized.any() and torch.equal(out[sized], chain[sized])  # formed again as one chain
    rest = chain.isfinite() & ~sized
    bound = 2 * (K + 2) * U * (x.abs().double() @ w.abs().double().T)
    assert ((out.double() - chain.double()).abs() <= bound)[rest].all()
