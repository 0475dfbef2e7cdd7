"""The product of floats whose operands are cut into bfloat16 pieces, at the ends of the range of operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


def rnd(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("M,N", [(3, 300), (40, 9000)])  # K split and not
@pytest.mark.parametrize("ex,ew", [(-118, 60), (-126, 90), (-138, 100), (60, -118), (90, -126), (-112, 50), (-30, 60), (75, -60)])
def test_small_operands_against_large_ones(M, N, ex, ew):
    """No bit of an operand is lost, down to the smallest: pieces of subnormal size would not hold it."""
    from dispec_b200.ops import gemm
    K = 512
    x, w = rnd((M, K), 1) * 2.0 ** ex, rnd((N, K), 2) * 2.0 ** ew
    out = gemm._split(x, w, None, None, torch.empty((M, N), device=DEV))
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # as in test_split_product_gpu.py, or where a result is formed as one chain, its K sums
    bound = torch.where(ref.abs() < 2.0 ** -59, 2.0 * K, 4 + 16 + K / 128 + 12) * U * size
    assert ((out.double() - ref).abs() <= bound).all()


def test_rows_of_very_different_sizes():
    """A row of tiny values among others, a matrix with a huge row: each result as if it were alone."""
    from dispec_b200.ops import gemm
    x, w = rnd((24, 1536), 3), rnd((640, 1536), 4)
    x[5] *= 2.0 ** -115
    x[7, ::2] *= 2.0 ** -120
    w[9] *= 2.0 ** 70
    w[11, 1::2] *= 2.0 ** -130
    out = gemm._split(x, w, None, None, torch.empty((24, 640), device=DEV))
    chain = gemm._simt(x, w, None, None, torch.empty((24, 640), device=DEV))
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    error = ((out.double() - ref).abs() / size).max()
    assert error <= (4 + 16 + 12 + 12) * U or error <= ((chain.double() - ref).abs() / size).max()


def test_products_that_underflow():
    """Results near the smallest numbers are those of the chain of FMAs."""
    from dispec_b200.ops import gemm
    for e in (-64, -70, -73, -74):
        x, w = rnd((8, 512), 5).abs() * 2.0 ** e, rnd((256, 512), 6).abs() * 2.0 ** e
        out, chain = (f(x, w, None, None, torch.empty((8, 256), device=DEV)) for f in (gemm._split, gemm._simt))
        assert torch.equal(out, chain) and (e < -73 or bool((out != 0).all()))


def test_rows_without_numbers_are_not_slow():
    """A result that is no number is formed again one by one; all of them together take no more than some ten times the
    product (rows of a step that hold nothing are computed with the others)."""
    from dispec_b200.ops import gemm
    x, w = rnd((264, 1536), 7), rnd((4096, 1536), 8)
    out = torch.empty((264, 4096), device=DEV)

    def ms(a):
        gemm._split(a, w, None, None, out)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        gemm._split(a, w, None, None, out)
        end.record()
        end.synchronize()
        return start.elapsed_time(end)

    usual = min(ms(x) for _ in range(5))
    assert ms(torch.full_like(x, float("nan"))) < 12 * usual and bool(out.isnan().all())
    x[100, 3] = float("nan")
    assert ms(x) < 3 * usual and bool(out[100].isnan().all()) and bool(out[99].isfinite().all())


@pytest.mark.parametrize("N,K", [(512, 1536), (2048, 1536), (3072, 2048), (4096, 4096), (8960, 1536), (14336, 2048)])
def test_few_rows_are_not_slower_than_the_chain(N, K):
    """A matrix goes to the same kernel for every number of rows, so that one row must not pay for many."""
    from dispec_b200.ops import gemm
    x, w = rnd((1, K), 9), rnd((N, K), 10)
    assert gemm.split_supported(w)
    out = torch.empty((1, N), device=DEV)

    def us(f):
        f(x, w, None, None, out)
        torch.cuda.synchronize()
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(20):
                f(x, w, None, None, out)
        times = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            graph.replay()
            end.record()
            end.synchronize()
            times.append(50 * start.elapsed_time(end))
        return min(times)

    assert us(gemm._split) < 1.25 * us(gemm._simt)


@pytest.mark.parametrize("K", [1536, 4096, 8960])
@pytest.mark.parametrize("kind", ["uniform", "lognormal", "squares", "half"])
def test_operands_of_one_sign(kind, K):
    """The tensor cores cut sums off, always towards zero: products of one sign must not add that up beyond what a chain of
    FMAs rounds."""
    from dispec_b200.ops import gemm
    g = torch.Generator(device=DEV).manual_seed(K)
    u = lambda s: torch.randn(s, generator=g, device=DEV)
    draw = {"uniform": lambda s: torch.rand(s, generator=g, device=DEV), "lognormal": lambda s: torch.exp(2 * u(s)),
            "squares": lambda s: u(s) ** 2, "half": lambda s: u(s).relu()}[kind]
    x, w = draw((48, K)), draw((512, K))
    ref = x.double() @ w.double().T
    error = lambda f: float((f(x, w, None, None, torch.empty((48, 512), device=DEV)).double() - ref).norm() / ref.norm())
    assert error(gemm._split) < error(gemm._simt)
