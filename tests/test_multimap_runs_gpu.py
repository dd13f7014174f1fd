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


@pytest.mark.parametrize("distinct,crowd", [(1500, 0), (1500, 300), (400_000, 0)])
def test_table_sized_by_the_distinct_keys(distinct, crowd):
    """Batches large enough for a table of the estimated number of keys; with `crowd` keys that all hash to one place,
    so that the small table is given up for a full-size one."""
    import b2co
    import torch
    rng = np.random.default_rng(distinct + crowd)
    n = (1 << 20) + 3
    keys = np.unique(rng.integers(0, 2**62, size=distinct, dtype=np.int64))
    if crowd:
        keys = np.concatenate([keys, fmix64_inverse((np.arange(1, crowd + 1, dtype=np.uint64) << np.uint64(40)) + np.uint64(77))])
    keys = keys[keys != -1]
    at = np.concatenate([np.arange(len(keys)), rng.integers(0, len(keys), size=n - len(keys))])
    v = rng.integers(0, 2**40, size=n, dtype=np.int64)
    m = b2co.StaticMultimap(n, -1, -1, key_dtype=torch.int64, value_dtype=torch.int64)
    assert m.Insert(b2co.pack_pairs(dev(keys[at]), dev(v))) == 0
    q = np.concatenate([keys, keys ^ np.int64(1 << 50)])
    counts = np.bincount(at, minlength=len(keys))
    total = int(counts.sum())
    assert m.Count(dev(keys)) == total
    ko = torch.zeros(total, dtype=torch.int64, device="cuda")
    vo = torch.zeros(total, dtype=torch.int64, device="cuda")
    assert m.Retrieve(dev(keys), ko, vo, total) == total
    order = np.lexsort((v, at))
    assert np.array_equal(ko.cpu().numpy(), keys[at[order]])
    assert np.array_equal(vo.cpu().numpy(), v[order])
    flags = torch.zeros(len(q), dtype=torch.uint8, device="cuda")
    m.Contains(dev(q), flags)
    assert np.array_equal(flags.cpu().numpy(), np.isin(q, keys).astype(np.uint8))
