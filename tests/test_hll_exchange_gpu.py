"""HyperLogLog Add where its CTAs exchange registers with the sketch during a batch (no exchange, one, two), into an
empty sketch and into one that holds keys already, from aligned and unaligned starts.  Registers are compared exactly."""
import numpy as np
import pytest

import oracle
from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bytes", [4, 8])
@pytest.mark.parametrize("precision,n", [(17, 1_500_000), (15, 11_000_003), (13, 4_000_001), (13, 12_000_005)])
def test_registers_after_exchanges(precision, n, key_bytes):
    import b2co
    import torch
    rng = np.random.default_rng(precision + n)
    kdt = np.int32 if key_bytes == 4 else np.int64
    keys = rng.integers(np.iinfo(kdt).min, np.iinfo(kdt).max, size=n, dtype=kdt)
    h = b2co.HyperLogLog(precision, key_dtype=torch.int32 if key_bytes == 4 else torch.int64)
    reg = np.zeros(1 << precision, np.uint8)
    kd = dev(keys)
    for lo, hi in [(0, n // 2), (n // 2 | 1, n)]:
        h.Add(kd[lo:hi])
        oracle.hll_add(reg, precision, keys[lo:hi])
        assert np.array_equal(h.registers(), reg)
