"""Working memory of the latent attention of prompts: what it takes, and what a refusal leaves behind."""
import pytest
import torch


def test_a_refusal_is_remembered_and_tried_again():
    from dispec_b200.cache.storage import CacheStorage
    s = CacheStorage([], 16, [], torch.float32, "cpu")
    assert s.room_beside(1 << 30)
    s.no_room_beside(1000)
    assert s.room_beside(999) and not s.room_beside(1000)
    s.no_room_beside(500)
    s.no_room_beside(2000)
    assert not s.room_beside(500) and s.room_beside(499)
    for _ in range(s.ROOM_RETRY):
        s.room_beside(500)
    assert s.room_beside(500)


def test_rows_are_allocated_in_few_sizes():
    from dispec_b200.ops import latent as LO
    rooms = [LO.expanded_room(n) for n in range(1, 200000)]
    assert all(n <= room <= max(n + 63, 1.25 * n) for n, room in enumerate(rooms, 1))
    assert len({r for r in rooms if r >= 1024}) <= 40
    # the gathered latents count as well
    assert LO.expanded_bytes([4], [1 << 16], 2, 64, 64, 64, 0) == 2 * (1 << 16) * (256 + 64 + 64)


@pytest.mark.parametrize("requests,stored,new,heads,width,rank,expanded", [
    (1, 0, 2, 12, 256, 512, True), (1, 1000, 2, 12, 256, 512, True), (1, 1000, 512, 12, 256, 512, True),
    (1, 8000, 2, 12, 256, 512, True), (4, 400, 16, 12, 256, 512, True), (2, 0, 1250, 12, 256, 512, True),
    (16, 0, 64, 12, 256, 512, True), (32, 1000, 2, 12, 256, 512, False), (32, 400, 16, 12, 256, 512, False),
    (32, 0, 2, 12, 256, 512, False), (32, 1000, 32, 12, 256, 512, True), (64, 1000, 8, 12, 256, 512, False),
    (1, 8000, 16, 4, 128, 128, True), (32, 1000, 64, 4, 128, 128, True), (16, 1000, 16, 32, 256, 512, False),
    (16, 400, 64, 32, 256, 512, True), (32, 0, 512, 32, 256, 512, True),
])
def test_which_side_of_the_rule(requests, stored, new, heads, width, rank, expanded):
    """Where both forms were measured and one was a tenth faster or more."""
    from dispec_b200.ops import latent as LO
    q, c = [new] * requests, [stored + new] * requests
    assert LO.expanded_is_faster(q, c, heads, width, rank, 0, 148) is expanded
    # a window bounds what a portion sees, and with it both estimates
    if stored + new > 500:
        assert LO.expanded_is_faster(q, c, heads, width, rank, stored + new, 148) is expanded

