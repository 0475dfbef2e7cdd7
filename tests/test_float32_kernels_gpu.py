"""The product and the attention on the FMA units alone, at the sizes where their tiles end."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24  # unit roundoff of float32


def rnd(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("M,N,K", [(1, 16, 4), (4, 17, 132), (5, 33, 128), (16, 15, 516), (17, 64, 36), (33, 65, 100),
                                   (64, 128, 64), (97, 129, 68), (129, 130, 32), (200, 31, 1000)])
def test_every_tile_gives_the_bits_of_one_chain(M, N, K):
    from dispec_b200.ops import gemm
    x, w, b, r = rnd((M, K), 1), rnd((N, K), 2), rnd((N,), 3), rnd((M, N), 4)
    ref = x.double() @ w.double().T + b.double() + r.double()
    # K products and sums, one bias and one residual, each rounded once
    bound = (K + 2) * U * (x.abs().double() @ w.abs().double().T + b.abs().double() + r.abs().double())
    first = None
    for tile in [-1] + list(range(10 if M <= 16 else 9)):
        out = gemm._simt(x, w, b, r, torch.full((M, N), float("nan"), device=DEV), tile)
        assert ((out.double() - ref).abs() <= bound).all(), tile
        first = out if first is None else first
        assert torch.equal(out, first), tile


@pytest.mark.parametrize("M,N,K,ld", [(3, 20, 5, 5), (7, 40, 64, 65), (40, 70, 33, 36)])
def test_rows_that_are_no_whole_pieces(M, N, K, ld):
    from dispec_b200.ops import gemm
    x = rnd((M, ld), 5)[:, ld - K:]  # an odd base as well
    w = rnd((N, K), 6)
    out = gemm.linear(x, w)
    bound = K * U * (x.abs().double() @ w.abs().double().T)
    assert ((out.double() - x.double() @ w.double().T).abs() <= bound).all()
    assert torch.equal(out[M // 2:M // 2 + 1], gemm.linear(x[M // 2:M // 2 + 1].contiguous(), w))


def seen(p, j, window, chunked, keep):
    if j > p:
        return False
    if not window or j < keep:
        return True
    return j // window == p // window if chunked else p - window < j


@pytest.mark.parametrize("H,G_heads,D,Dv,page,window,chunked,keep,sink", [
    (6, 1, 128, 128, 16, 0, False, 0, None),     # five tokens of six heads a block
    (3, 3, 4, 8, 8, 0, False, 0, "learned"),     # the smallest heads; 32 tokens of one head
    (40, 1, 32, 64, 16, 0, False, 0, None),      # more heads than a block has rows
    (12, 2, 48, 128, 32, 70, False, 0, "zero"),  # a window that ends inside tiles
    (8, 4, 64, 36, 16, 64, True, 0, None),       # chunks as long as a tile
    (4, 2, 100, 32, 8, 33, False, 5, "learned"),  # kept first keys, in the window's tiles or far from them
])
def test_attention_of_runs(H, G_heads, D, Dv, page, window, chunked, keep, sink):
    from dispec_b200.ops import attention as A
    from dispec_b200.ops import library as L
    spans = [(130, 1), (1, 1), (0, 75), (190, 40), (64, 2)]  # (stored, new) of each sequence
    T, S, most = sum(n for _, n in spans), len(spans), max(a + n for a, n in spans)
    pages = -(-most // page)
    kp, vp = (torch.full((S * pages + 1, G_heads, page, w), float("nan"), device=DEV) for w in (D, Dv))
    table = torch.full((S, pages), -1, dtype=torch.int32)
    q, out = rnd((T, H * D), 7), torch.full((T, H * Dv), float("nan"), device=DEV)
    zs = rnd((H,), 8) if sink == "learned" else None
    scale, G = D ** -0.5, H // G_heads
    positions, seqs, ref, free, row = [], [], [], S * pages, 0
    for s, (a, n) in enumerate(spans):
        k, v = rnd((a + n, G_heads, D), 20 + s), rnd((a + n, G_heads, Dv), 40 + s)
        for j in range(a + n):
            if table[s, j // page] < 0:
                free -= 1
                table[s, j // page] = free
            kp[table[s, j // page], :, j % page], vp[table[s, j // page], :, j % page] = k[j], v[j]
        for p in range(a, a + n):
            keys = [j for j in range(p + 1) if seen(p, j, window, chunked, keep)]
            x = q[row].view(G_heads, G, D).double()
            sc = torch.einsum("hgd,jhd->hgj", x, k[keys].double()) * scale
            if sink:
                z = (zs if zs is not None else torch.zeros(H, device=DEV)).double().view(G_heads, G, 1)
                sc = torch.cat([sc, z], -1)
            wts = torch.softmax(sc, -1)[..., :len(keys)]
            ref.append(torch.einsum("hgj,jhv->hgv", wts, v[keys].double()).reshape(-1))
            positions.append(p)
            seqs.append(s)
            row += 1
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    A.paged_attention_generic(q, H * D, kp, vp, table.to(DEV), i32(positions), i32(seqs), out, H, G_heads, D, window, scale,
                              sink=sink is not None, chunked=chunked, sink_values=zs, keep_first=keep)
    L.raise_on_device_error("attention")
    # scores of |q||k| scale ~ 6 at most with D rounded terms, expf within two units, sums of at most 230 weights
    tol = (D + 2 * 230 + 40) * U * 8
    assert (out.double() - torch.stack(ref)).abs().max() <= tol
    # the last key of the third sequence is no number: only its own row may change
    last = 74
    vp[table[2, last // page], :, last % page] = float("nan")
    again = torch.full_like(out, float("nan"))
    A.paged_attention_generic(q, H * D, kp, vp, table.to(DEV), i32(positions), i32(seqs), again, H, G_heads, D, window, scale,
                              sink=sink is not None, chunked=chunked, sink_values=zs, keep_first=keep)
    mine = 2 + last
    keepers = [i for i in range(T) if i != mine]
    assert torch.equal(again[keepers], out[keepers]) and again[mine].isnan().all()


@pytest.mark.parametrize("H,G_heads,D,window,chunked,keep,sink", [
    (12, 2, 128, 0, False, 0, False),   # one token: 8 rows on 32 lanes, five tokens: 32 rows on 16 lanes
    (4, 4, 64, 0, False, 0, True),      # up to 8 tokens on 32 lanes
    (9, 1, 32, 70, False, 0, False),    # always on 16 lanes
    (8, 2, 48, 33, False, 5, True),
    (6, 2, 16, 64, True, 0, False),
])
def test_attention_of_a_token_does_not_depend_on_its_portion(H, G_heads, D, window, chunked, keep, sink):
    """Every token of a portion alone, in pairs, and with the portion cut elsewhere: the same bits."""
    from dispec_b200.ops import attention as A
    n, first, page = 300, 130, 16
    kp, vp = (rnd((n // page + 1, G_heads, page, D), s) for s in (31, 32))
    kp *= 3.0  # weights of very different sizes
    vp[3, :, 2, 1] = float("inf")  # and a value that a weight which is merely small does not hide
    table = torch.arange(kp.shape[0], dtype=torch.int32, device=DEV)[None]
    q, z = rnd((n - first, H * D), 33), rnd((H,), 34)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(lo, hi):
        out = torch.full((hi - lo, H * D), 7.0, device=DEV)
        return A.paged_attention_generic(q[lo:hi], H * D, kp, vp, table, i32(list(range(first + lo, first + hi))),
                                         i32([0] * (hi - lo)), out, H, G_heads, D, window, D ** -0.5, sink=sink, chunked=chunked,
                                         sink_values=z if sink else None, keep_first=keep)

    whole = run(0, n - first).view(torch.int32)
    for cut in (1, 2, 7, 50):
        parts = torch.cat([run(a, min(n - first, a + cut)) for a in range(0, n - first, cut)])
        assert torch.equal(parts.view(torch.int32), whole), cut


@pytest.mark.parametrize("dtype,hidden", [(torch.float32, h) for h in (8, 512, 768, 772, 1536)]
                         + [(torch.bfloat16, h) for h in (8, 256, 1024, 1032, 1536, 1544, 2048, 2056, 3072, 3080)])
def test_rms_norm_of_a_row_does_not_depend_on_the_others(dtype, hidden):
    from dispec_b200 import ops
    x, w, delta = rnd((2500, hidden), 41).to(dtype), rnd((hidden,), 42).to(dtype), rnd((2500, hidden), 43).to(dtype)
    whole, summed = ops.rms_norm(x, w, 1e-6), ops.rms_norm(x, w, 1e-6, delta=delta)
    for n in (1, 3, 592, 1775, 1776):
        assert torch.equal(ops.rms_norm(x[:n].contiguous(), w, 1e-6), whole[:n]), n
        assert torch.equal(ops.rms_norm(x[:n].contiguous(), w, 1e-6, delta=delta[:n].contiguous()), summed[:n]), n


@pytest.mark.parametrize("M,N,K", [(1, 3, 5), (7, 64, 17), (64, 65, 33), (65, 130, 15), (3, 1000, 515)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_bfloat16_widths_that_are_no_multiple_of_eight(M, N, K, out_dtype):
    from dispec_b200.ops import gemm
    x, w, b = (rnd(shape, s).bfloat16() for shape, s in (((M, K), 51), ((N, K), 52), ((N,), 53)))
    r = rnd((M, N), 54).to(out_dtype)
    out = gemm.linear(x, w, b, residual=r, out_dtype=out_dtype, backend="simt")
    ref = x.double() @ w.double().T + b.double() + r.double()
    bound = (K + 2) * U * (x.abs().double() @ w.abs().double().T + b.abs().double() + r.abs().double())
    if out_dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * (ref.abs() + bound)  # the result is rounded once
    assert ((out.double() - ref).abs() <= bound).all()
    one = gemm.linear(x[M // 2:M // 2 + 1].contiguous(), w, b, residual=r[M // 2:M // 2 + 1].contiguous(), out_dtype=out_dtype,
                      backend="simt")
    assert torch.equal(out[M // 2:M // 2 + 1], one)
