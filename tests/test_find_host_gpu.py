"""Host-buffer Find from and into pinned and pageable memory, around the sizes where its chunks change.  Exact."""
import numpy as np
import pytest

from helpers import make_pairs, unique_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,vb", [(8, 8), (4, 4)])
def test_pinned_and_pageable_buffers(kb, vb):
    import b2co
    import torch
    kd, vd = {4: torch.int32, 8: torch.int64}[kb], {4: torch.int32, 8: torch.int64}[vb]
    rng = np.random.default_rng(kb)
    keys = unique_keys(rng, 200_000, kb)
    vals = unique_keys(rng, 200_000, vb)
    t = b2co.StaticMap(500_000, -1, -1, key_dtype=kd, value_dtype=vd)
    assert t.Insert(make_pairs(keys[:100_000], vals[:100_000])) == 0
    for n in (1, 131_071, 131_072, 131_073, 524_289, (1 << 22) - 1, (1 << 22) + 1):
        at = rng.integers(0, len(keys), size=n)
        q, want = keys[at], np.where(at < 100_000, vals[at], -1).astype(vals.dtype)
        pq, po = b2co.pinned(n, q.dtype), b2co.pinned(n, want.dtype)
        pq[:] = q
        for src in (pq, np.array(q)):
            for dst in (po, np.empty(n, want.dtype)):
                dst[:] = 7
                t.FindHost(src, dst)
                assert np.array_equal(dst, want), n
