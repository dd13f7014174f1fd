"""StaticMultimap's index on both sides of the line from 2,048 to 4,096 partitions, with batches that give every block
of the routing pass several tiles.  The expected groups are sorted on the GPU by torch; every result is exact."""
import pytest

from helpers import torch_dt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 4), (8, 4)])
@pytest.mark.parametrize("n", [1 << 23, (1 << 23) + 1, (1 << 24) + 1])
def test_partitions(kb, vb, n):
    import b2co
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n + kb)
    d = n // 4
    ids = torch.randint(0, d, (n,), device="cuda", generator=g)

    def key_of(i):  # an odd multiplier: distinct keys of distinct numbers, in [0, 2^31)
        return ((i * 0x2C1B3C6D) & 0x7FFFFFFF).to(torch_dt(kb))

    keys = key_of(ids)
    vals = torch.randint(-2**31, 2**31 - 1, (n,), device="cuda", generator=g)
    vals = torch.where(vals == -1, torch.zeros_like(vals), vals)
    if vb == 8:
        vals = vals * 0x100000001  # both halves of the word in use, the order kept
        vals = torch.where(vals == -1, torch.zeros_like(vals), vals)
    m = b2co.StaticMultimap(n, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb))
    assert m.Insert(b2co.pack_pairs(keys, vals.to(torch_dt(vb)))) == 0
    # all present keys, each once, in a random order, with as many absent ones
    present = torch.unique(ids)
    q_ids = torch.cat([present, present + d])[torch.randperm(2 * len(present), device="cuda", generator=g)]
    q = key_of(q_ids)
    flags = torch.full((len(q),), 9, dtype=torch.uint8, device="cuda")
    m.Contains(q, flags)
    assert torch.equal(flags, (q_ids < d).to(torch.uint8))
    assert m.Count(q) == n
    ko = torch.zeros(n, dtype=torch_dt(kb), device="cuda")
    vo = torch.zeros(n, dtype=torch_dt(vb), device="cuda")
    assert m.Retrieve(q, ko, vo, n) == n
    # expected: the pairs by (place of their key's query, value)
    rank = torch.empty(2 * d, dtype=torch.int64, device="cuda")
    rank[q_ids] = torch.arange(len(q), device="cuda")
    order = torch.argsort(vals)
    order = order[torch.argsort(rank[ids[order]], stable=True)]
    assert torch.equal(ko, keys[order])
    assert torch.equal(vo, vals.to(torch_dt(vb))[order])
