"""Groups whose items lie in large tables take the tiled kernels by default.  A large table among small ones (empty,
full and too small for their keys), around chunk and pass ends; values are known by construction, so all is exact."""
import numpy as np
import pytest

from helpers import dev, make_pairs, torch_dt, unique_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bucket", [1, 2, 5])
@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 4), (4, 0), (8, 4)])
def test_large_table_among_small_ones(kb, vb, bucket):
    import b2co
    import torch
    rng = np.random.default_rng(kb * 10 + vb + bucket)
    big = (340 << 20) // b2co.slot_bytes(kb, vb)
    counts = np.array([300, 0, 150_001, 33, 0, 511, 1, 700])
    caps = np.array([600, 10, big, 40, 1, 700, 1, 350])  # the last one has half as many slots as keys
    g = b2co.TableGroup(caps, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb) if vb else None,
                        bucket_size=bucket)
    if bucket > 1:
        assert g.find_shape()[0] == 2
    keys = unique_keys(rng, int(counts.sum()), kb)
    vals = unique_keys(rng, len(keys), vb) if vb else None
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    room = [g.table_capacity(t) for t in range(len(caps))]
    lost = sum(max(0, int(c) - r) for c, r in zip(counts, room))
    pairs = make_pairs(keys, vals)
    assert g.Insert(pairs, dev(off)) == lost
    assert g.Insert(pairs, dev(off)) == len(keys)
    out = torch.zeros(len(keys), dtype=torch_dt(vb or kb), device="cuda")
    flags = torch.zeros(len(keys), dtype=torch.uint8, device="cuda")
    want = vals if vb else keys
    for find in (lambda o, c: g.Find(dev(keys), dev(off), o, contains=c),
                 lambda o, c: g.Find(dev(keys), dev(off), o, contains=c, graph=True)):
        out.fill_(5)
        find(out, False)
        got = out.cpu().numpy()
        hit = got == want
        assert hit[: off[7]].all() and hit[off[7]:].sum() == 700 - lost and (got[~hit] == -1).all()
        flags.fill_(9)
        find(flags, True)
        assert np.array_equal(flags.cpu().numpy(), hit.astype(np.uint8))
    g.Clear()
    g.Find(dev(keys), dev(off), flags, contains=True)
    assert not flags.any()


def test_few_items_in_a_large_slab():
    """The same for a few items in many tables that together are past L2."""
    import b2co
    import torch
    rng = np.random.default_rng(3)
    g = b2co.TableGroup(np.full(300, 100_000), -1, -1, key_dtype=torch.int64, value_dtype=torch.int64)
    counts = rng.integers(0, 300, size=300)
    keys = unique_keys(rng, int(counts.sum()), 8)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    pairs = make_pairs(keys, np.arange(len(keys)))
    assert g.Insert(pairs, dev(off)) == 0
    assert g.Insert(pairs, dev(off)) == len(keys)
    out = torch.zeros(len(keys), dtype=torch.int64, device="cuda")
    g.Find(dev(keys), dev(off), out)
    assert np.array_equal(out.cpu().numpy(), np.arange(len(keys)))
