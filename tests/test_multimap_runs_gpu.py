"""StaticMultimap's grouped index at the edges of its sorts: runs that one thread, one warp and one block sort, runs
left to the radix sort, tiles whose runs do not fit shared memory, and a batch whose last pair is refused.  Values are
integers, so every result is compared exactly."""
import numpy as np
import pytest

from helpers import NP_DT, dev, torch_dt

pytestmark = pytest.mark.gpu

RUNS = {
    "edges": [1, 2, 24, 25, 31, 32, 33, 255, 256, 257, 4095, 4096],
    "radix": [4097, 9000, 1, 70001],
    "full_tiles": [24] * 700 + [23] * 40,
    "single": [1] * 2000,
    "one_run": [3],
}


@pytest.mark.parametrize("kb,vb", [(4, 4), (4, 8), (8, 4), (8, 8)])
@pytest.mark.parametrize("name", sorted(RUNS))
def test_runs_come_back_ascending(kb, vb, name):
    import b2co
    import torch
    rng = np.random.default_rng(kb * 100 + vb)
    lengths = np.array(RUNS[name])
    keys = (np.arange(len(lengths)) * 7919 + 5).astype(NP_DT[kb])
    info = np.iinfo(NP_DT[vb])
    k = np.repeat(keys, lengths)
    v = rng.integers(info.min + 1, info.max, size=len(k), dtype=NP_DT[vb], endpoint=True)
    v[v == -1] = 0
    v[: len(v) // 3] %= 5  # repeated values among them
    order = rng.permutation(len(k))
    k, v = k[order], v[order]
    m = b2co.StaticMultimap(len(k) + 3, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb))
    assert m.Insert(b2co.pack_pairs(dev(k), dev(v))) == 0
    # a batch with one reserved pair changes nothing
    bad = b2co.pack_pairs(dev(np.array([1, 2, -1], NP_DT[kb])), dev(np.array([1, 2, 3], NP_DT[vb])))
    with pytest.raises(b2co.InvalidArgument):
        m.Insert(bad)
    assert m.Size() == len(k)
    q = np.concatenate([keys[::-1], np.array([3], NP_DT[kb])])  # 3 is absent
    at = np.lexsort((v, k))
    ks, vs = k[at], v[at]
    lo, hi = np.searchsorted(ks, q, "left"), np.searchsorted(ks, q, "right")
    total = int((hi - lo).sum())
    assert m.Count(dev(q)) == total
    ko = torch.zeros(total, dtype=torch_dt(kb), device="cuda")
    vo = torch.zeros(total, dtype=torch_dt(vb), device="cuda")
    assert m.Retrieve(dev(q), ko, vo, total) == total
    assert np.array_equal(ko.cpu().numpy(), np.concatenate([ks[a:b] for a, b in zip(lo, hi)]))
    assert np.array_equal(vo.cpu().numpy(), np.concatenate([vs[a:b] for a, b in zip(lo, hi)]))
    first = torch.zeros(len(q), dtype=torch_dt(vb), device="cuda")
    m.Find(dev(q), first)
    assert np.array_equal(first.cpu().numpy(), np.where(hi > lo, vs[np.minimum(lo, len(vs) - 1)], -1).astype(NP_DT[vb]))


def fmix64_inverse(h):
    """Keys whose MurmurHash3 64-bit finalizer is h (each step of it undone)."""
    m = (1 << 64) - 1
    x = h.astype(object)
    inv1 = pow(0xC4CEB9FE1A85EC53, -1, 1 << 64)
    inv2 = pow(0xFF51AFD7ED558CCD, -1, 1 << 64)
    x = x ^ (x >> 33)
    x = (x * inv1) & m
    x = x ^ (x >> 33)
    x = (x * inv2) & m
    x = x ^ (x >> 33)
    return np.array([int(v) for v in x], dtype=np.uint64).view(np.int64)


@pytest.mark.parametrize("kb,vb", [(4, 4), (4, 8), (8, 4), (8, 8)])
@pytest.mark.parametrize("distinct,crowd,heavy", [
    (1500, 0, 0),        # too few keys for partitions of like size
    (1500, 300, 0),      # and too many of them in one place of the small table
    (400_000, 0, 0),     # by partitions
    (400_000, 300, 0),   # one partition's part of the table cannot hold its keys
    (400_000, 0, 1400),  # a key with a large share of its partition
    (400_000, 0, 9000),  # a partition too large for one block
    (1_000_000, 0, 0),
])
def test_batches_large_enough_to_be_surveyed(distinct, crowd, heavy, kb, vb):
    import b2co
    import torch
    if crowd and kb == 4:
        pytest.skip("the crowded keys are made for the 64-bit hash")
    rng = np.random.default_rng(distinct + crowd + heavy)
    n = (1 << 20) + 3
    ki, vi = np.iinfo(NP_DT[kb]), np.iinfo(NP_DT[vb])
    keys = np.unique(rng.integers(0, ki.max // 2, size=distinct, dtype=NP_DT[kb]))
    if crowd:
        keys = np.concatenate([keys, fmix64_inverse((np.uint64(77) << np.uint64(50)) + np.arange(crowd, dtype=np.uint64))])
        keys = np.unique(keys[keys != -1])
    at = np.concatenate([np.arange(len(keys)), np.full(heavy, 5), rng.integers(0, len(keys), size=n - len(keys) - heavy)])
    at = rng.permutation(at)
    v = rng.integers(vi.min + 1, vi.max, size=n, dtype=NP_DT[vb])
    v[v == -1] = 0
    m = b2co.StaticMultimap(n, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb))
    assert m.Insert(b2co.pack_pairs(dev(keys[at]), dev(v))) == 0
    assert m.Count(dev(keys)) == n
    ko = torch.zeros(n, dtype=torch_dt(kb), device="cuda")
    vo = torch.zeros(n, dtype=torch_dt(vb), device="cuda")
    assert m.Retrieve(dev(keys), ko, vo, n) == n
    order = np.lexsort((v, at))
    assert np.array_equal(ko.cpu().numpy(), keys[at[order]])
    assert np.array_equal(vo.cpu().numpy(), v[order])
    q = np.concatenate([keys, keys ^ NP_DT[kb](ki.max // 2 + 1)])
    flags = torch.zeros(len(q), dtype=torch.uint8, device="cuda")
    m.Contains(dev(q), flags)
    assert np.array_equal(flags.cpu().numpy(), np.isin(q, keys).astype(np.uint8))
