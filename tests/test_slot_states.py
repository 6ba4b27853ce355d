"""States that start at zero lie behind one another in one tensor, by size: a taken slot is cleared in every site and nowhere else,
and every site's state is contiguous and begins at a multiple of 512 bytes."""

import pytest
import torch

from tandemllm_b200.cache.manager import CacheManager
from tandemllm_b200.parts.base import PagedNeed, SlotNeed


@pytest.mark.parametrize("slots", [1, 3, 7])
def test_a_taken_slot_is_cleared_in_every_site_and_nowhere_else(slots):
    shapes = [(2, 5), (2, 5), (3,), (2, 5), (128,), (1,)]
    needs = [SlotNeed(s, torch.float32) for s in shapes] + [(PagedNeed(1, 16), SlotNeed((2, 5), torch.float32)), SlotNeed((1,), torch.int32, init=-1)]
    cache = CacheManager(needs, num_pages=2, max_requests=slots, device="cpu")
    states = [c.state for c in cache.site_cache[:6]] + [cache.site_cache[6][1].state, cache.site_cache[7].state]
    base = {}
    for s, shape in zip(states, shapes + [(2, 5), (1,)]):
        assert tuple(s.shape) == (slots, *shape) and s.is_contiguous()
        assert (s.storage_offset() * s.element_size()) % 512 == 0
        s.fill_(3)
        base.setdefault(s.untyped_storage().data_ptr(), []).append(s)
    assert sorted(len(v) for v in base.values()) == [1, 1, 1, 1, 4]
    slot = cache.admit("a")
    for s in states:
        assert (s[slot] == (-1 if s.dtype == torch.int32 else 0)).all()
        assert (s[[i for i in range(slots) if i != slot]] == 3).all()
