"""DynamicMap over several submaps against a dict (the passes that mark older submaps' keys and the lookups that ask
the newest submap first), and the counts that synchronous inserts report, also from several threads at once.
Everything is compared exactly."""
import threading

import numpy as np
import pytest

from helpers import NP_DT, dev, torch_dt, unique_keys

pytestmark = pytest.mark.gpu


def pairs(k, v):
    import b2co
    return b2co.pack_pairs(dev(k), dev(v))


@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (4, 8), (8, 4)])
@pytest.mark.parametrize("big", [False, True])  # big: submaps above the sector kernels' size
def test_updates_and_lookups_over_submaps(kb, vb, big):
    import b2co
    import torch
    rng = np.random.default_rng(kb * 10 + vb)
    first = 30_000_000 if big else 60_000
    m = b2co.DynamicMap(first, -1, -1, -2, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb))
    n = 120_001
    keys = unique_keys(rng, n, kb)
    vals = rng.integers(0, 2**30, size=n).astype(NP_DT[vb])
    d = {}
    at = 0
    for size, reserve in ((15_000, 0), (40_003, 20_000_000), (64_998, 60_000_000)):
        if big:  # small submaps grow by themselves (a batch is more than the room left), large ones are added here
            m.Reserve(reserve)
        k, v = keys[at:at + size], vals[at:at + size]
        assert m.Insert(pairs(k, v)) == size
        d.update(zip(k.tolist(), v.tolist()))
        at += size
    assert m.Size() == n and m.NumSubmaps() > 1
    # present keys are not inserted again, wherever they live; duplicates of a new key count once
    extra = unique_keys(rng, 3000, kb, lo=2**30 if kb == 4 else 2**62, hi=2**31 - 2 if kb == 4 else 2**63 - 2)
    mix = np.concatenate([keys[::7], extra, extra[:500], np.array([-1], NP_DT[kb])])
    v = (mix.astype(np.int64) % 1000003).astype(NP_DT[vb])  # duplicates carry the same payload
    assert m.Insert(pairs(mix, v)) == len(extra)
    d.update(zip(extra.tolist(), (extra.astype(np.int64) % 1000003).tolist()))
    # updates of old and new keys alike
    more = unique_keys(rng, 2000, kb, lo=2**29 + 1 if kb == 4 else 2**61, hi=2**30 - 1 if kb == 4 else 2**62 - 1)
    more = more[~np.isin(more, keys)]
    up = np.concatenate([keys[3::5], extra[::3], more])
    rng.shuffle(up)
    uv = rng.integers(0, 2**30, size=len(up)).astype(NP_DT[vb])
    assert m.InsertOrAssign(pairs(up, uv)) == len(more)
    d.update(zip(up.tolist(), uv.tolist()))
    assert m.Size() == len(d)
    absent = np.arange(5, 5 + 4000).astype(NP_DT[kb])
    absent = absent[~np.isin(absent, np.array(list(d), dtype=NP_DT[kb]))]
    q = np.concatenate([np.array(list(d), dtype=NP_DT[kb]), absent])
    rng.shuffle(q)
    want = np.array([d.get(x, -1) for x in q.tolist()]).astype(NP_DT[vb])
    out = torch.full((len(q),), 3, dtype=torch_dt(vb), device="cuda")
    m.Find(dev(q), out)
    assert np.array_equal(out.cpu().numpy(), want)
    flags = torch.full((len(q),), 3, dtype=torch.uint8, device="cuda")
    m.Contains(dev(q), flags)
    assert np.array_equal(flags.cpu().numpy(), np.array([x in d for x in q.tolist()]).astype(np.uint8))


def test_oldest_submap_answers_first():
    """A caller that breaks the unique-keys promise has a key in two submaps: the older one's payload is found, unless
    it is the empty payload."""
    import b2co
    import torch
    m = b2co.DynamicMap(60_000, -1, -1, -2, key_dtype=torch.int64, value_dtype=torch.int64)
    k = np.arange(1, 10_001, dtype=np.int64)
    v = k * 3
    v[::10] = -1  # stored with the empty payload
    assert m.Insert(pairs(k, v)) == len(k)
    assert m.Insert(pairs(k + 1_000_000, k), mode=m.kExactDedup) == len(k)
    m.Insert(pairs(np.arange(2_000_000, 2_040_000, dtype=np.int64), np.arange(40_000, dtype=np.int64)))
    assert m.NumSubmaps() >= 2
    m.Insert(pairs(k, k * 5), mode=m.kAppendUnique)
    out = torch.empty(len(k), dtype=torch.int64, device="cuda")
    m.Find(dev(k), out)
    want = k * 3
    want[::10] = k[::10] * 5
    assert np.array_equal(out.cpu().numpy(), want)


def test_counts_of_concurrent_inserts():
    """Synchronous inserts into one table from several threads and streams: each call's counts are its own."""
    import b2co
    import torch
    t = b2co.StaticMap(1 << 21, -1, -1, key_dtype=torch.int64, value_dtype=torch.int64)
    rounds, threads = 20, 4
    wrong = []

    def work(w):
        s = torch.cuda.Stream()
        base = w * 10_000_000
        for r in range(rounds):
            n = 1000 + 977 * ((w + r) % 9)
            k = np.arange(base, base + n, dtype=np.int64) + 5
            base += n
            p = pairs(np.concatenate([k, k[: 100 * w + r]]), np.concatenate([k, k[: 100 * w + r]]))
            torch.cuda.synchronize()
            if t.Insert(p, stream=s) != 100 * w + r:
                wrong.append(("insert", w, r))
            if t.InsertOrAssign(p, stream=s, with_assigned=True) != (0, n + 100 * w + r):
                wrong.append(("assign", w, r))

    ts = [threading.Thread(target=work, args=(w,)) for w in range(threads)]
    for x in ts:
        x.start()
    for x in ts:
        x.join()
    assert not wrong
