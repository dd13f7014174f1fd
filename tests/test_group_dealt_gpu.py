"""Group batches large enough to have their chunks dealt by a counter: Insert and Find of a few more items than the line
between the two, on several streams with more launches in flight than there are counters, and captured (where chunks go
by warp number).  Keys are unique, so every result is known, and is compared with one launch per table as well."""
import numpy as np
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kdt,vdt", [("int32", "int32"), ("int64", "int64")])
def test_dealt_batches(kdt, vdt):
    import b2co
    import torch
    kdt, vdt = getattr(torch, kdt), getattr(torch, vdt)
    rng = np.random.default_rng(17)
    n = (1 << 25) + 77
    cuts = np.sort(rng.choice(n, size=250, replace=False))
    off = np.concatenate([[0], cuts, [n]]).astype(np.uint64)
    sizes = np.diff(off).astype(np.int64)
    d_off = dev(off.astype(np.int64))
    i = torch.arange(n, device="cuda")
    keys = (i * 2654435761) % (1 << 30)  # unique: an odd factor modulo a power of two
    values = (keys * 7 + 3) % (1 << 30)
    g = b2co.TableGroup(2 * sizes + 8, -1, -1, key_dtype=kdt, value_dtype=vdt)
    pairs = b2co.pack_pairs(keys.to(kdt), values.to(vdt))
    assert g.Insert(pairs, d_off) == 0
    assert g.Insert(pairs, d_off) == n  # all there already
    miss = i % 3 == 1
    q = torch.where(miss, keys + (1 << 30), keys).to(kdt)
    expected = torch.where(miss, torch.full_like(values, -1), values).to(vdt)
    out = torch.empty(n, dtype=vdt, device="cuda")
    g.FindPerTable(q, off, out)
    assert torch.equal(out, expected)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    outs = [torch.zeros(n, dtype=vdt, device="cuda") for _ in range(3)]
    flags = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for r in range(21):
        g.Find(q, d_off, outs[r % 3], stream=streams[r % 3])
    g.Find(q, d_off, flags, contains=True, stream=streams[0])
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, expected)
    assert torch.equal(flags.bool(), ~miss)
    out.zero_()
    g.Find(q, d_off, out, graph=True)
    torch.cuda.synchronize()
    assert torch.equal(out, expected)
