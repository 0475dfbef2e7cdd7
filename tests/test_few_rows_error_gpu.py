"""32-bit results of the few-row product: how far the sums of operands of one sign, which the tensor cores cut off on one
side, lie from 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


@pytest.mark.parametrize("M,parts", [(1, 4), (8, 4), (16, 4), (17, 2), (32, 2), (64, 2)])
def test_sums_of_one_sign(M, parts):
    from dispec_b200.ops import gemm
    N, K = 20480, 4096  # more blocks of W than SMs: K is not split
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = (torch.rand(s, generator=g, device=DEV).to(torch.bfloat16) for s in ((M, K), (N, K)))
    out = gemm._stream(x, w, None, None, torch.empty((M, N), device=DEV))
    ref = torch.cat([x.double() @ p.double().T for p in w.split(4096)], 1)
    mean = float(((out.double() - ref) / ref).mean())
    # a chain of n sums of 16 products, each cut off by half a last place (2 U of the sum so far, which is half the last
    # one on average) or less: n U / 2 and less; half as much again, and the products' own alignment and the parts' sum
    steps = K / 16 / parts
    assert abs(mean) < (0.75 * steps + 8) * U
