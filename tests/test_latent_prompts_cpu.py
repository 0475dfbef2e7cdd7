"""Working memory of the latent attention of prompts: what it takes, and what a refusal leaves behind."""
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
