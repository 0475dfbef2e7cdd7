"""The 32-bit attention of a token in runs of 32 rows (a long portion) and of 16 (a short one): the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,G_heads,D", [(32, 8, 64), (16, 16, 32), (24, 4, 128)])
def test_long_and_short_portions(H, G_heads, D):
    from dispec_b200.ops import attention as A
    n, page = 1300, 16
    rnd = lambda *s, seed: torch.randn(*s, generator=torch.Generator().manual_seed(seed)).to(DEV)
    kp, vp = (rnd(n // page + 1, G_heads, page, D, seed=s) for s in (1, 2))
    table = torch.arange(kp.shape[0], dtype=torch.int32, device=DEV)[None]
    q = rnd(n, H * D, seed=3)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)

    def run(lo, hi):
        out = torch.empty(hi - lo, H * D, device=DEV)
        return A.paged_attention_generic(q[lo:hi], H * D, kp, vp, table, i32(list(range(lo, hi))), i32([0] * (hi - lo)), out, H,
                                         G_heads, D, 0, D ** -0.5)

    # the whole is more blocks than two an SM, a part is not
    assert (n // (32 // (H // G_heads)) + 1) * G_heads > 2 * 148 >= (90 // (32 // (H // G_heads)) + 1) * G_heads
    whole = run(0, n)
    for a, b in ((0, 90), (611, 700), (n - 1, n)):
        assert torch.equal(run(a, b), whole[a:b]), (a, b)
