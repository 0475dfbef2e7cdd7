"""The 32-bit attention in runs of 16 and of 32 rows, on 256 and on 128 threads: a token has the same bits in all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,KVH,D,kernels", [(40, 2, 128, 1), (34, 2, 64, 2), (24, 8, 96, 2), (32, 32, 64, 3), (12, 2, 128, 3)])
def test_requests_of_one_token_and_portions(H, KVH, D, kernels):
    from dispec_b200.ops import attention as A, library as L
    page, single, portion = 16, 160, 900
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    contexts = [5 + (17 * i) % 190 for i in range(single)]
    pages = -(-portion // page)
    # all requests on the same pages: their keys are alike, their queries are not
    kp, vp = (rnd(pages, KVH, page, D, seed=s) for s in (1, 2))
    table = torch.arange(pages, dtype=torch.int32, device=DEV)[None].repeat(single + 1, 1)
    positions = i32([n - 1 for n in contexts] + list(range(portion)))
    request = i32(list(range(single)) + [single] * portion)
    q = rnd(single + portion, H * D, seed=3)
    used = set()

    def run(lo, hi, num_single):
        out = torch.full((hi - lo, H * D), float("nan"), device=DEV)
        used.add(L.core().dsp_attn_rows_choice(hi - lo, num_single, 0, H, KVH, D, D, 148))
        return A.paged_attention_generic(q[lo:hi], H * D, kp, vp, table, positions[lo:hi], request[lo:hi], out, H, KVH, D, 0,
                                         D ** -0.5, num_single=num_single)

    whole = run(0, single + portion, single)
    for lo, hi, n in ((0, single, single), (0, single, 0), (0, 1, 1), (7, 9, 2), (single, single + portion, 0),
                      (single, single + 40, 0), (single + 611, single + 700, 0), (single + portion - 1, single + portion, 1)):
        assert torch.equal(run(lo, hi, n), whole[lo:hi]), (lo, hi, n)
    assert len(used) == kernels
    # against 64 bits
    x = q.double().view(-1, KVH, H // KVH, D)
    k, v = (t.permute(1, 0, 2, 3).reshape(KVH, -1, D).double() for t in (kp, vp))
    s = torch.einsum("tkgd,knd->tkgn", x, k) * D ** -0.5
    hidden = torch.arange(s.shape[-1], device=DEV)[None, :] > positions[:, None].long()
    s = s.masked_fill(hidden[:, None, None, :], float("-inf"))
    want = torch.einsum("tkgn,knd->tkgd", s.softmax(-1), v).reshape(single + portion, H * D)
    assert (whole.double() - want).abs().max() < 1e-5  # weights of 32 bits over values of magnitude 1
