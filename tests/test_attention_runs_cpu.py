"""How the 32-bit attention cuts its work: runs of 16 rows only where a group of heads fits one and all their blocks run at
once, 128 threads only where blocks are many."""
import pytest


@pytest.mark.parametrize("T,singles,longest,H,KVH,D,kernel", [
    (1, 1, 1000, 12, 2, 128, 0), (264, 4, 330, 12, 2, 128, 0), (8, 8, 0, 64, 4, 64, 0), (128, 128, 600, 64, 4, 64, 0),
    # more than 16 heads on a KV head: 16 rows would walk all keys twice
    (1, 1, 600, 40, 2, 128, 1), (64, 64, 600, 40, 2, 128, 1), (128, 0, 0, 40, 2, 128, 1), (1, 1, 9, 32, 1, 64, 1), (1, 1, 9, 48, 1, 128, 1),
    # twice as many blocks of 16 rows would no longer run at once
    (400, 0, 1000, 12, 2, 128, 1), (400, 0, 0, 12, 2, 128, 1), (264, 0, 864, 32, 8, 128, 1), (2000, 0, 2000, 12, 2, 128, 1),
    # a prompt from its first token on: the longest block bounds it
    (400, 0, 400, 12, 2, 128, 0), (500, 0, 500, 12, 2, 128, 0),
    # many single tokens, many small blocks
    (64, 64, 600, 32, 8, 128, 2), (256, 256, 600, 12, 2, 128, 2), (16, 16, 0, 16, 16, 128, 2), (800, 0, 1400, 16, 8, 64, 2),
])
def test_the_choice(T, singles, longest, H, KVH, D, kernel):
    from dispec_b200.ops import library
    assert library.core().dsp_attn_rows_choice(T, singles, longest, H, KVH, D, D, 148) == kernel
