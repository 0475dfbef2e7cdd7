"""The norm of a sum four elements at a time, xIELU by rows, the RMS norm a warp a row."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


def rnd(shape, seed, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


@pytest.mark.parametrize("width", [4, 508, 1536, 2048, 2052, 4096, 4100, 6])
@pytest.mark.parametrize("x_dtype,off", [(torch.float32, 0), (torch.bfloat16, 0), (torch.float32, 1)])
def test_sum_norm(width, x_dtype, off):
    from dispec_b200.ops import norm32
    n, alpha, eps = 5, 1.75, 1e-5
    x = rnd((n, width + 4), 5, 1.0, x_dtype)[:, off:off + width]
    delta, w = rnd((n, width + 4), 6)[:, off:off + width], rnd((width,), 7) + 1.0
    rows = torch.tensor([4, 0, 4, 2], dtype=torch.int32, device=DEV)
    for d, r in ((delta, None), (None, None), (delta, rows)):
        y32, y16 = norm32.sum_norm(x, w, eps, alpha=alpha, delta=d, rows=r, out_dtype=torch.bfloat16)[:2]
        s = alpha * x.double() + (d.double() if d is not None else 0.0)
        if r is not None:
            s = s[r.long()]
        want = s / torch.sqrt((s * s).mean(-1, keepdim=True) + eps) * w.double()
        # two roundings in the sum, a mean of `width` squares, a root, a quotient and two products
        tol = (width + 10) * U * (want.abs() + (alpha * x.double().abs().max() + delta.double().abs().max()) * U)
        assert ((y32.double() - want).abs() <= tol + 4 * U).all()
        assert torch.equal(y16, y32.to(torch.bfloat16))


@pytest.mark.parametrize("rows,cols", [(1, 4), (3, 2048), (2, 2052), (5, 8960), (2500, 60), (4, 66),
                                       # one group a thread and four, and their last stretches
                                       (2368, 512), (2369, 512), (64, 1536), (700, 2044), (800, 2052), (5000, 132)])
def test_xielu_rows(rows, cols):
    from dispec_b200.ops import norm32
    z = rnd((rows, cols + 4), 14, 3.0)[:, :cols]
    p, q = 0.4, -0.7
    y = norm32.xielu(z, torch.tensor([p, q], device=DEV), torch.bfloat16).double()
    sp = lambda v: torch.log1p(torch.exp(torch.tensor(v, dtype=torch.float64, device=DEV)))
    v = z.double()
    want = torch.where(v > 0, sp(p) * v * v, (0.5 + sp(q)) * (torch.expm1(v.clamp(max=0)) - v)) + 0.5 * v
    # rounded to bfloat16 once (2^-8 with what 32 bits leave open); the two terms below zero nearly cancel
    assert ((y - want).abs() <= 2.0 ** -8 * want.abs() + 32 * U * (1 + v.abs())).all()


@pytest.mark.parametrize("n,hidden", [(592, 1536), (593, 8), (600, 1032), (595, 1544), (700, 768), (591, 1536),
                                      # a warp a row: each share of a row that a lane can have, full and not, and beyond it
                                      (1776, 8), (1777, 1024), (1780, 1032), (1800, 1536), (1776, 1544), (1779, 2048),
                                      (1790, 2056), (1801, 3072), (1776, 3080), (1775, 1536)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rms_norm_of_many_rows(n, hidden, dtype):
    from dispec_b200 import ops
    x, w, delta = rnd((n, hidden), 11, 2.0, dtype), (1.0 + rnd((hidden,), 12, 0.2)).to(dtype), rnd((n, hidden), 13, 1.0, dtype)
    rows = torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV)

    def want(v):
        unit = (v.double() / torch.sqrt((v.double() ** 2).mean(-1, keepdim=True) + 1e-6)).to(dtype)
        return w.double() * unit.double()

    # a unit row may round the other way, which is one unit in its last place (2^-7 of it at most in bfloat16), and the
    # product is rounded once (2^-8)
    tol = (2.0 ** -7 + 2.0 ** -8 if dtype == torch.bfloat16 else (hidden + 10) * U)
    close = lambda y, v: ((y.double() - want(v)).abs() <= tol * (want(v).abs() + 1e-3)).all()
    assert close(ops.rms_norm(x, w, 1e-6), x)
    assert torch.equal(ops.rms_norm(x, w, 1e-6, rows=rows), ops.rms_norm(x, w, 1e-6).flip(0))
    total = (x.double() + delta.double()).to(dtype)
    y = x.clone()
    out = ops.rms_norm(y, w, 1e-6, delta=delta, write_back=True)
    assert torch.equal(y, total) and close(out, total)
