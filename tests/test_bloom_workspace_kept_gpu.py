"""A routed Bloom Add's workspace is kept with the filter: a batch of several rounds settles it, a captured Add replays
whatever Adds came after it, and where memory is short what could be had is kept.  Words are compared exactly with those
of a filter that takes no workspace."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONGEST = (1 << 27) // 8 * 9  # keys of the longest round


def filters(blocks):
    import b2co
    import torch
    plain, routed = (b2co.BloomFilter(blocks, key_dtype=torch.int32) for _ in range(2))
    plain.set_add_mode(b2co.BLOOM_ADD_ATOMIC)
    routed.set_add_mode(b2co.BLOOM_ADD_PARTITIONED)
    return plain, routed


def keys_of(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-2**31, 2**31 - 1, (n,), dtype=torch.int32, device="cuda", generator=g)


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def capture(f, keys):
    import torch
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        f.AddAsync(keys, stream=s)
    torch.cuda.synchronize()
    return g


def same(a, b):
    import torch
    torch.cuda.synchronize()
    return np.array_equal(a.words(), b.words())


def test_a_batch_of_two_rounds_settles_the_workspace():
    plain, routed = filters(1 << 22)
    keys = keys_of(LONGEST + 10_000_001, 1)
    few = keys[5:5 + (1 << 22)]
    routed.Add(keys)  # two rounds
    plain.Add(keys)
    assert same(plain, routed)
    g = capture(routed, few)
    left = free_bytes()
    for n in (1 << 27, LONGEST):  # one round each, longer than those two
        routed.Clear()
        plain.Clear()
        routed.Add(keys[:n])
        plain.Add(keys[:n])
        assert same(plain, routed)
        assert free_bytes() == left
    routed.Clear()
    plain.Clear()
    g.replay()
    plain.Add(few)
    assert same(plain, routed)


def test_a_captured_add_outlives_a_larger_one():
    import torch
    plain, routed = filters(1 << 20)
    few, many = keys_of(3_000_001, 2), keys_of(30_000_001, 3)
    routed.Add(few)
    g = capture(routed, few)
    routed.Add(many)  # wants a larger workspace
    other = torch.full((1 << 25,), -1, dtype=torch.int32, device="cuda")  # takes what has been given back
    for _ in range(2):
        routed.Clear()
        plain.Clear()
        g.replay()
        plain.Add(few)
        assert same(plain, routed)
    assert bool((other == -1).all())


def test_what_little_memory_gave_is_kept():
    import torch
    plain, routed = filters(1 << 20)
    n = (1 << 25) + 5
    keys = keys_of(n, 4)
    plain.Add(keys)
    routed.Add(keys[:1000])
    torch.cuda.empty_cache()
    hog = torch.empty(max(0, free_bytes() - (256 << 20)), dtype=torch.uint8, device="cuda")
    routed.Add(keys)  # shorter rounds
    assert same(plain, routed)
    routed.Clear()
    g = capture(routed, keys)  # a capture cannot allocate
    left = free_bytes()
    routed.Add(keys)
    assert free_bytes() == left
    assert same(plain, routed)
    routed.Clear()
    g.replay()
    assert same(plain, routed)
    del hog
    torch.cuda.empty_cache()
