"""Latent attention of portions of prompts on expanded keys and values, alone and beside single tokens."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def turned(x, pos, freq, layout, mag):
    """x [..., r] at position pos."""
    n = freq.shape[0]
    c, s = torch.cos(pos * freq) * mag, torch.sin(pos * freq) * mag
    y = x.clone()
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if layout == "interleaved" else (x[..., :n], x[..., n:2 * n])
    a, b = u * c - v * s, v * c + u * s
    if layout == "interleaved":
        y[..., 0:2 * n:2], y[..., 1:2 * n:2] = a, b
    else:
        y[..., :n], y[..., n:2 * n] = a, b
    return y


def setting(spans, H, R, d, dv, page, seed):
    """spans: (stored, new) of each sequence, single tokens first."""
    g = torch.Generator().manual_seed(seed)
    bf = lambda *shape, s=1.0: (torch.randn(*shape, generator=g) * s).bfloat16()
    lens, q_lens = [a + n for a, n in spans], [n for _, n in spans]
    pages = [-(-n // page) for n in lens]
    order = torch.randperm(sum(pages) + 2, generator=g)[:sum(pages)].tolist()
    tables = torch.full((len(spans), max(pages)), -1, dtype=torch.int32)
    c_pool = torch.full((sum(pages) + 2, 1, page, R), float("nan")).bfloat16()
    r_pool = torch.full((sum(pages) + 2, 1, page, 64), float("nan")).bfloat16()
    c, kr, at = [], [], 0
    for s, n in enumerate(lens):
        c.append(bf(n, R))
        kr.append(bf(n, 64))
        for j in range(pages[s]):
            tables[s, j] = order[at]
            m = min(page, n - j * page)
            c_pool[order[at], 0, :m], r_pool[order[at], 0, :m] = c[s][j * page:j * page + m], kr[s][j * page:j * page + m]
            at += 1
    T = sum(q_lens)
    tiles = [(s, a) for s, n in enumerate(q_lens) for a in range(0, n, 128)]
    starts = [0]
    for n in q_lens:
        starts.append(starts[-1] + n)
    n_dec = sum(n == 1 for n in q_lens)
    ctx = SimpleNamespace(attention_tiles={128: (i32([s for s, _ in tiles]), i32([a for _, a in tiles]), len(tiles))},
                          q_start=i32(starts), ctx_len=i32(lens), num_decode_seqs=n_dec, host_q_len=q_lens, host_ctx_len=lens)
    return SimpleNamespace(ctx=ctx, tables=tables, c_pool=c_pool.to(DEV), r_pool=r_pool.to(DEV), c=c, kr=kr, lens=lens,
                           q_lens=q_lens, starts=starts, n_dec=n_dec, T=T, q=bf(T, H * (d + 64), s=1.5),
                           w=bf(H * (d + dv), R, s=R ** -0.5), gate=torch.randn(T, H * dv + 3, generator=g),
                           sink=torch.randn(H, generator=g) + 1.0)


@pytest.mark.parametrize("spans,H,R,d,dv,page,window,layout,rot,sink,gate", [
    ([(0, 2)], 1, 64, 128, 128, 16, 0, "interleaved", 64, False, False),
    ([(0, 128), (0, 129)], 3, 512, 128, 128, 16, 0, "interleaved", 64, True, False),
    ([(70, 1), (3, 1), (65, 63), (0, 300), (511, 2)], 2, 104, 128, 128, 16, 0, "halves", 32, True, True),
    ([(0, 64), (64, 64)], 12, 96, 64, 128, 32, 0, "interleaved", 0, False, True),
    ([(200, 1), (130, 150), (640, 17)], 2, 72, 128, 64, 8, 40, "halves", 64, True, True),
    ([(1000, 90)], 2, 64, 64, 64, 64, 256, "interleaved", 64, False, False),
])
def test_expanded_keys_and_values(spans, H, R, d, dv, page, window, layout, rot, sink, gate):
    from dispec_b200.ops import latent as LO
    from dispec_b200.ops import library
    x = setting(spans, H, R, d, dv, page, 11)
    if window:  # pages that every query has left behind are given back
        for s, n in enumerate(x.lens):
            gone = max(0, n - x.q_lens[s] - window + 1) // page
            x.c_pool[x.tables[s, :gone].long().to(DEV)] = float("nan")
            x.tables[s, :gone] = -1
    scale, mag = 0.09, 1.2
    freq = (100.0 ** (-torch.arange(rot // 2).double() / 32)).float()
    out = torch.full((x.T, H * dv + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
    mine = out[:, :H * dv]
    assert LO.prompt_supported(d, 64, dv, R)
    LO.latent_attention_prompts(x.ctx, x.q.to(DEV), d + 64, d, freq.to(DEV) if rot else None, rot, x.c_pool, x.r_pool,
                                x.tables.to(DEV), x.w.to(DEV), mine, H, d, dv, scale, layout=layout, magnitude=mag,
                                window=window, sink=x.sink.to(DEV) if sink else None,
                                gate=x.gate.to(DEV)[:, 3:] if gate else None)
    assert library.device_error() == 0
    assert out[:, H * dv:].isnan().all() and out[:x.n_dec].isnan().all()
    got, w = mine.double().cpu(), x.w.double()
    for s, (n, ql) in enumerate(zip(x.lens, x.q_lens)):
        if ql == 1:
            continue
        # keys and values as the kernel reads them: rounded to bfloat16 once
        kv = (x.c[s].double() @ w.T).bfloat16().double()
        k, v = kv[:, :H * d].view(n, H, d), kv[:, H * d:].view(n, H, dv)
        for t in range(ql):
            p, row = n - ql + t, x.starts[s] + t
            lo = max(0, p - window + 1) if window else 0
            q = x.q[row].view(H, d + 64)
            qr = turned(q[:, d:].double(), p, freq.double(), layout, mag).bfloat16().double()
            sc = (torch.einsum("hd,jhd->hj", q[:, :d].double(), k[lo:p + 1]) + qr @ x.kr[s][lo:p + 1].double().T) * scale
            if sink:
                sc = torch.cat([sc, x.sink[:, None].double()], -1)
            wts = torch.softmax(sc, -1)[:, :p + 1 - lo]
            want = torch.einsum("hj,jhv->hv", wts, v[lo:p + 1]).reshape(-1)
            if gate:
                want = want * torch.sigmoid(x.gate[row, 3:].double())
            # weights are rounded to bfloat16 (2^-9 each), as are the turned queries and the result
            assert (got[row] - want).abs().max() < 0.02 * max(1.0, want.abs().max().item()), (s, t)


def test_a_bad_page_is_hidden_and_reported():
    from dispec_b200.ops import latent as LO
    from dispec_b200.ops import library
    H, R, d, dv, page = 2, 64, 128, 128, 16
    x = setting([(100, 30)], H, R, d, dv, page, 5)
    run = lambda tables: LO.latent_attention_prompts(
        x.ctx, x.q.to(DEV), d + 64, d, None, 0, x.c_pool, x.r_pool, tables.to(DEV), x.w.to(DEV), out, H, d, dv, 0.05)
    library.device_error()
    out = torch.empty((30, H * dv), dtype=torch.bfloat16, device=DEV)
    broken = x.tables.clone()
    broken[0, 2] = x.c_pool.shape[0]
    run(broken)
    assert library.device_error() == 1
    kv = (x.c[0].double() @ x.w.double().T).bfloat16().double()
    k, v = kv[:, :H * d].view(130, H, d), kv[:, H * d:].view(130, H, dv)
    keys = [j for j in range(130) if j // page != 2]
    q = x.q[29].view(H, d + 64).double()
    sc = (torch.einsum("hd,jhd->hj", q[:, :d], k[keys]) + q[:, d:] @ x.kr[0][keys].double().T) * 0.05
    want = torch.einsum("hj,jhv->hv", torch.softmax(sc, -1), v[keys]).reshape(-1)
    assert (out[29].double().cpu() - want).abs().max() < 0.02 * max(1.0, want.abs().max().item())


def small_model_logits(expand):
    """Logits of two steps of a small model with portions of prompts and single tokens."""
    from dispec_b200 import load_model_config
    from dispec_b200.engine import ModelRunner, SeqEntry
    from dispec_b200.ops import latent as LO
    from dispec_b200.weights import load_random_model
    layer = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 256},
             "mixer": {"heads": 4, "dim": 64, "rot_dim": 64, "vdim": 64, "kv_rank": 64, "q_rank": 96, "scale": 0.1,
                       "rot": {"base": 1e4, "dims": 64}}}
    cfg = {"architecture": "Puludra", "vocab": 300, "width": 128, "postln_alpha": 1.5, "norm": {"eps": 1e-6},
           "layers": [layer, layer]}
    model = load_random_model(load_model_config(cfg), 1, 0.1, "bfloat16", DEV)
    g = torch.Generator().manual_seed(1)
    ids = [torch.randint(0, 300, (400,), generator=g).tolist() for _ in range(3)]
    most, LO.PROMPT_MAX_BYTES = LO.PROMPT_MAX_BYTES, 1 << 30 if expand else 0
    try:
        r = ModelRunner(model, page_size=16, num_pages=100, max_num_seqs=3)
        for i in range(3):
            r.admit(i)
        out = [r.step([SeqEntry(0, ids[0][:150], 0, [149]), SeqEntry(1, ids[1][:33], 0, [32])]).clone()]
        out.append(r.step([SeqEntry(0, ids[0][150:151], 150, [0]), SeqEntry(1, ids[1][33:200], 33, [166, 1]),
                           SeqEntry(2, ids[2][:70], 0, [69])]).clone())
        r.check_device()
        return torch.cat(out)
    finally:
        LO.PROMPT_MAX_BYTES = most


def test_mixers_of_both_kinds_agree():
    """A small model's logits with its portions on expanded keys and on the latents."""
    a, b = small_model_logits(True), small_model_logits(False)
    assert ((a - b).norm() / b.norm()).item() < 0.02 and not torch.equal(a, b)


def test_without_room_for_the_expanded_rows(monkeypatch):
    from dispec_b200.ops import latent as LO

    def no_room(*args, **kwargs):
        raise torch.OutOfMemoryError("no room")

    a = small_model_logits(True)
    monkeypatch.setattr(LO, "latent_attention_prompts", no_room)
    assert torch.equal(small_model_logits(True), small_model_logits(False)) and not torch.equal(a, small_model_logits(True))


@pytest.mark.parametrize("first", [1, 4])
def test_output_columns_that_begin_anywhere(monkeypatch, first):
    """Heads whose output rows do not begin on 16 bytes (columns of a wider row): on the latents, as they were."""
    from dispec_b200.parts.latent_attention import LatentAttention
    heads = LatentAttention.heads

    def shifted(self, ctx, z, cache, state, out):
        wide = torch.empty((out.shape[0], out.shape[1] + 8), dtype=out.dtype, device=out.device)
        heads(self, ctx, z, cache, state, wide[:, first:first + out.shape[1]])
        out.copy_(wide[:, first:first + out.shape[1]])

    monkeypatch.setattr(LatentAttention, "heads", shifted)
    a, b = small_model_logits(True), small_model_logits(False)
    assert torch.equal(a, b) and a.isfinite().all()


def test_a_refusal_is_asked_for_once(monkeypatch):
    """Two layers and two steps without room: the expanded rows are asked for in the first layer of the first step."""
    from dispec_b200.ops import latent as LO
    asked = []

    def no_room(*args, **kwargs):
        asked.append(1)
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(LO, "latent_attention_prompts", no_room)
    assert torch.equal(small_model_logits(True), small_model_logits(False)) and len(asked) == 1
