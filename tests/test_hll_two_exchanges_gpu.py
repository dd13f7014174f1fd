"""HyperLogLog Add where a batch is long enough for its CTAs to exchange registers with the sketch twice (four keys a
register and CTA or more), from unaligned starts and into a sketch that holds keys already.  Registers are exact."""
import numpy as np
import pytest

import oracle
from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bytes", [4, 8])
def test_registers_after_two_exchanges(key_bytes):
    import b2co
    import torch
    precision, n = 13, 24_000_005
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (n // 2 // (2 * sms)) >> precision >= 4  # two CTAs an SM
    rng = np.random.default_rng(key_bytes)
    kdt = np.int32 if key_bytes == 4 else np.int64
    keys = rng.integers(np.iinfo(kdt).min, np.iinfo(kdt).max, size=n, dtype=kdt)
    h = b2co.HyperLogLog(precision, key_dtype=torch.int32 if key_bytes == 4 else torch.int64)
    reg = np.zeros(1 << precision, np.uint8)
    kd = dev(keys)
    for lo, hi in [(0, n // 2), (n // 2 | 1, n)]:
        h.Add(kd[lo:hi])
        oracle.hll_add(reg, precision, keys[lo:hi])
        assert np.array_equal(h.registers(), reg)
