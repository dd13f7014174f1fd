"""A routed Bloom Add that finds no room for its longest round's records takes shorter rounds."""
import numpy as np
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


def test_add_with_little_memory_left():
    import b2co
    import torch
    n = (1 << 25) + 5
    keys = dev(np.random.default_rng(3).integers(0, 2**62, size=n, dtype=np.int64))
    plain, routed = (b2co.BloomFilter(1 << 20, key_dtype=torch.int64) for _ in range(2))
    plain.set_add_mode(b2co.BLOOM_ADD_ATOMIC)
    plain.Add(keys)
    routed.set_add_mode(b2co.BLOOM_ADD_PARTITIONED)
    routed.Add(keys[:1000])
    torch.cuda.empty_cache()
    hog = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (256 << 20)), dtype=torch.uint8, device="cuda")
    routed.Add(keys)  # a round for all of them wants more than what is left
    del hog
    torch.cuda.empty_cache()
    assert np.array_equal(plain.words(), routed.words())
