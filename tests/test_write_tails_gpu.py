"""The ends of the write kernels' batches: pairs that are left when a warp has no full pass any more walk on lane by
lane, in tables that are nearly full (long walks, lost and whole cycles), for every slot width, window and write
kernel.  Results are compared with values known by construction."""
import numpy as np
import pytest

from helpers import LAYOUTS, dev, make_pairs, torch_dt, unique_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bucket", [1, 2, 5, 8])
@pytest.mark.parametrize("kb,vb", LAYOUTS)
@pytest.mark.parametrize("shape", [(0, 0), (1, 1), (4, 1)])
def test_last_pairs_of_a_batch(kb, vb, bucket, shape):
    import b2co
    import torch
    rng = np.random.default_rng(kb * 100 + vb * 10 + bucket)
    kw = dict(bucket_size=bucket, probing=b2co.PROBE_DOUBLE, hash_kind=b2co.HASH_XXH32)
    t = (b2co.StaticMap(3000, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb), **kw) if vb else
         b2co.StaticSet(3000, -1, key_dtype=torch_dt(kb), **kw))
    t.set_write_shape(*shape)
    cap = t.Capacity()
    keys = unique_keys(rng, cap + 70, kb)
    vals = unique_keys(rng, cap + 70, vb) if vb else keys
    pairs = lambda sel, v=None: make_pairs(keys[sel], (vals if v is None else v)[sel] if vb else None)
    n0 = int(0.95 * cap)
    at = 0
    while at < n0:  # batches that end anywhere in a warp
        m = min(int(rng.integers(1, 200)), n0 - at)
        assert t.Insert(pairs(np.arange(at, at + m))) == 0
        at += m
    present = np.arange(n0)

    def race(sel, want_found, want_inserted):
        found = torch.full((len(sel),), 5, dtype=torch_dt(vb or kb), device="cuda")
        inserted = torch.full((len(sel),), 5, dtype=torch.uint8, device="cuda")
        t.InsertAndFind(pairs(sel), found, inserted, mode=b2co.IAF_RACE)
        assert np.array_equal(found.cpu().numpy(), want_found)
        assert np.array_equal(inserted.cpu().numpy(), want_inserted)

    for n in (1, 31, 33, 300):
        sel = rng.choice(present, size=n)
        race(sel, vals[sel], np.zeros(n, np.uint8))
        assert t.Insert(pairs(sel)) == n
    new = np.arange(n0, n0 + 40)
    both = rng.permutation(np.concatenate([new, rng.choice(present, size=60)]))
    race(both, vals[both], (both >= n0).astype(np.uint8))
    if vb:
        vals2 = vals.copy()
        vals2[: n0 + 40] = vals[: n0 + 40][::-1]
        sel = np.arange(n0 + 40)
        assert t.InsertOrAssign(pairs(sel, vals2), with_assigned=True) == (0, n0 + 40)
        out = torch.zeros(n0 + 40, dtype=torch_dt(vb), device="cuda")
        t.Find(dev(keys[sel]), out)
        assert np.array_equal(out.cpu().numpy(), vals2[sel])
        vals = vals2
    # fill the table: the pairs that find no slot have gone round their whole cycle
    rest = np.arange(n0 + 40, cap + 70)
    assert t.Insert(pairs(rest, vals)) == 70
    flags = torch.zeros(len(rest), dtype=torch.uint8, device="cuda")
    t.Contains(dev(keys[rest]), flags)
    inside = flags.cpu().numpy().astype(bool)
    assert inside.sum() == len(rest) - 70
    out_of = rest[~inside]
    found = torch.zeros(70, dtype=torch_dt(vb or kb), device="cuda")
    inserted = torch.ones(70, dtype=torch.uint8, device="cuda")
    t.InsertAndFind(pairs(out_of, vals), found, inserted, mode=b2co.IAF_RACE)
    assert (found.cpu().numpy() == -1).all() and not inserted.any()
