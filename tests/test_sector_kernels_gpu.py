"""The one-lane sector kernels and the staged lookups around the sizes where they can go wrong: batches that end
inside a warp's pass, a block or a stage, streams that start off a 16-byte boundary, stencils, nearly full tables
(keys that probe on through the queue, and whole probe cycles), and the table and batch sizes where the default
changes from one kernel to the other.  Everything is compared exactly with the oracle or with values known by
construction."""
import numpy as np
import pytest

import oracle
from helpers import LAYOUTS, NP_DT, dev, make_pairs, miss_keys, oracle_table, torch_dt, unique_keys

pytestmark = pytest.mark.gpu

# shapes: the default, one lane a key, and the staged kernels
SHAPES = {"auto": None, "sector": (1, 1), "staged_2x1": (2, 1, False, False, False, True),
          "staged_4x2": (4, 2, False, False, False, True)}


def new_table(kb, vb, slots, bucket=5, probing=None, hash_kind=None):
    import b2co
    kw = dict(bucket_size=bucket, probing=b2co.PROBE_DOUBLE if probing is None else probing,
              hash_kind=b2co.HASH_XXH32 if hash_kind is None else hash_kind)
    if vb == 0:
        return b2co.StaticSet(slots, -1, key_dtype=torch_dt(kb), **kw)
    return b2co.StaticMap(slots, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb), **kw)


@pytest.mark.parametrize("bucket", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("kb,vb", LAYOUTS)
def test_nearly_full_table_ragged_batches(kb, vb, bucket):
    import b2co
    import torch
    rng = np.random.default_rng(kb * 100 + vb * 10 + bucket)
    t = new_table(kb, vb, 6000, bucket)
    cap = t.Capacity()
    # more keys than slots: the table ends full, and what finds no slot has gone round its whole cycle
    keys = unique_keys(rng, cap + 40, kb)
    vals = None if vb == 0 else unique_keys(rng, cap + 40, vb)
    o = oracle_table(t, kb, vb, bucket, oracle.PROBE_DOUBLE, oracle.HASH_XXH32)
    n0 = int(0.97 * cap)
    assert t.Insert(make_pairs(keys[:n0], None if vb == 0 else vals[:n0])) == 0
    assert o.insert(keys[:n0], None if vb == 0 else vals[:n0]) == 0
    q = np.concatenate([keys[:n0], miss_keys(rng, 700, kb)])
    rng.shuffle(q)
    expected, _ = o.find(q)
    for n in (1, 2, 31, 32, 33, 63, 64, 65, 257, 1023, 1024, 1025, len(q)):
        for start in (0, 1, 3):  # streams on and off a 16-byte boundary
            sub = dev(q)[start:start + n]
            m = len(sub)
            want = expected[start:start + m]
            stencil = (rng.random(m) < 0.5).astype(np.uint8)
            for name, shape in SHAPES.items():
                t.set_find_shape(*(shape or (0, 0)))
                out = torch.full((m,), 7, dtype=torch_dt(vb or kb), device="cuda")
                t.Find(sub, out)
                assert np.array_equal(out.cpu().numpy(), want), (name, n, start)
                flags = torch.full((m,), 9, dtype=torch.uint8, device="cuda")
                t.Contains(sub, flags)
                assert np.array_equal(flags.cpu().numpy(), (want != -1).astype(np.uint8)), (name, n, start)
                t.FindIf(sub, dev(stencil), out)
                assert np.array_equal(out.cpu().numpy(), np.where(stencil, want, -1)), (name, n, start)
    t.set_find_shape(0, 0)
    # fill it up: every slot taken, 40 or more keys without one
    rest = make_pairs(keys[n0:], None if vb == 0 else vals[n0:])
    assert t.Insert(rest) == len(keys) - cap
    out = torch.empty(700, dtype=torch_dt(vb or kb), device="cuda")
    t.Find(dev(miss_keys(rng, 700, kb)), out)  # a whole cycle each
    assert (out.cpu().numpy() == -1).all()
    if vb:
        assert t.InsertOrAssign(rest, with_assigned=True) == (len(keys) - cap, cap - n0)


@pytest.mark.parametrize("kb,vb,slots", [(8, 8, 15_500_000), (4, 4, 30_000_000), (4, 0, 70_000_000)])
def test_default_changes_with_batch_and_table(kb, vb, slots):
    """Tables above the sector kernels' size: batches on both sides of the batch rule, every kernel alike."""
    import b2co
    import torch
    t = new_table(kb, vb, slots)
    n = 3_000_001
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ids = torch.arange(n, dtype=torch.int64, device="cuda")
    keys = ((ids * 0x2C1B3C6D) & 0x7FFFFFFF).to(torch_dt(kb))  # an odd multiplier: distinct 31-bit keys
    vals = None if vb == 0 else (ids ^ 0x155555).to(torch_dt(vb))
    for shape in ((0, 0), (1, 1), (4, 1)):
        t.Clear()
        t.set_write_shape(*shape)
        assert t.Insert(keys if vb == 0 else b2co.pack_pairs(keys, vals)) == 0
        for m in (98_303, 98_304, 98_305, 131_072, 262_145, n):
            at = torch.randint(0, 2 * n, (m,), device="cuda", generator=g)
            q = ((at * 0x2C1B3C6D) & 0x7FFFFFFF).to(torch_dt(kb))
            payload = q if vb == 0 else (at ^ 0x155555).to(torch_dt(vb))
            want = torch.where(at < n, payload, torch.full_like(payload, -1))
            for name, sh in SHAPES.items():
                t.set_find_shape(*(sh or (0, 0)))
                out = torch.empty_like(want)
                t.Find(q, out)
                assert torch.equal(out, want), (shape, name, m)
                out.zero_()
                t.Find(q[1:], out[1:])
                assert torch.equal(out[1:], want[1:]), (shape, name, m, "off a boundary")


@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (4, 0), (8, 4)])
@pytest.mark.parametrize("count", [1, 3, 40, 1100])
def test_group_chunks(kb, vb, count):
    """Groups whose tables end inside a chunk, are empty, or are smaller than a pass; full tables among them."""
    import b2co
    import torch
    rng = np.random.default_rng(count * 10 + kb + vb)
    sizes = rng.integers(0, 90, size=count) if count > 3 else rng.integers(500, 9000, size=count)
    sizes[rng.random(count) < 0.2] = 0 if count > 3 else 300
    caps = np.maximum(sizes * 5 // 4, 1)
    g = b2co.TableGroup(caps, -1, -1, key_dtype=torch_dt(kb), value_dtype=torch_dt(vb) if vb else None)
    keys = unique_keys(rng, max(int(sizes.sum()), 1), kb)[: int(sizes.sum())]
    vals = np.arange(len(keys)).astype(NP_DT[vb]) if vb else None
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pairs = make_pairs(keys, vals)
    assert g.Insert(pairs, dev(off)) == 0
    assert g.Insert(pairs, dev(off)) == len(keys)  # every pair is present now
    # every table is asked its own keys and as many of the next table's
    q, want, qoff = [], [], [0]
    for t in range(count):
        own = np.arange(off[t], off[t + 1])
        other = np.arange(off[(t + 1) % count], off[(t + 1) % count + 1])
        at = np.concatenate([own, other])
        hit = np.concatenate([np.ones(len(own), bool), np.zeros(len(other), bool)])
        if count == 1:
            hit[:] = True
        order = rng.permutation(len(at))
        at, hit = at[order], hit[order]
        q.append(keys[at])
        want.append(np.where(hit, (vals if vb else keys)[at], -1))
        qoff.append(qoff[-1] + len(at))
    q = np.concatenate(q).astype(NP_DT[kb])
    want = np.concatenate(want).astype(NP_DT[vb or kb])
    for shape in ((1, 1, 0), (1, 1, 64), (2, 1, 0), (2, 2, 0), (4, 2, 128)):
        g.set_find_shape(*shape)
        out = torch.full((len(q),), 5, dtype=torch_dt(vb or kb), device="cuda")
        g.Find(dev(q), dev(np.array(qoff)), out)
        assert np.array_equal(out.cpu().numpy(), want), shape
        flags = torch.full((len(q),), 5, dtype=torch.uint8, device="cuda")
        g.Find(dev(q), dev(np.array(qoff)), flags, contains=True)
        assert np.array_equal(flags.cpu().numpy(), (want != -1).astype(np.uint8)), shape
