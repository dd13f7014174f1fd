"""StaticMultimap's index under keys that are made to fill a part of its table, or all of it, to the last slot: the
table must be built again at full size, and a lookup of an absent key must end.  The rules themselves run on the CPU
(tests/cpp/run_probe_test.cpp); the GPU cases compare every result exactly."""
import os
import subprocess

import numpy as np
import pytest

from helpers import dev

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
M64 = (1 << 64) - 1


def test_probe_rules_end_and_refuse(tmp_path):
    exe = str(tmp_path / "run_probe_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                    os.path.join(REPO, "ops-collections_b200", "csrc"),
                    os.path.join(REPO, "tests", "cpp", "run_probe_test.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    assert "run probe test ok" in r.stdout


def fmix64(k, seed=0):
    """MurmurHash3's 64-bit finalizer of k ^ seed."""
    k = k.view(np.uint64) ^ np.uint64(seed)
    k = (k ^ (k >> np.uint64(33))) * np.uint64(0xFF51AFD7ED558CCD)
    k = (k ^ (k >> np.uint64(33))) * np.uint64(0xC4CEB9FE1A85EC53)
    return k ^ (k >> np.uint64(33))


def fmix64_inverse(h):
    """The keys (int64) whose fmix64 is h."""
    h = h ^ (h >> np.uint64(33))
    h = h * np.uint64(pow(0xC4CEB9FE1A85EC53, -1, 1 << 64))
    h = h ^ (h >> np.uint64(33))
    h = h * np.uint64(pow(0xFF51AFD7ED558CCD, -1, 1 << 64))
    return (h ^ (h >> np.uint64(33))).view(np.int64)


def test_hash_and_inverse():
    h = np.random.default_rng(1).integers(0, M64, size=1000, dtype=np.uint64)
    assert np.array_equal(fmix64(fmix64_inverse(h)), h)


def full_region(rng):
    """400,000 random keys, and in one of 2,048 partitions a key for each of its 512 slots and no other."""
    part = np.uint64(77)
    keys = np.unique(rng.integers(0, 2**62, size=400_000, dtype=np.int64))
    keys = keys[(fmix64(keys) >> np.uint64(53)) != part]
    crafted = fmix64_inverse((part << np.uint64(53)) | (np.arange(512, dtype=np.uint64) << np.uint64(44)) | np.uint64(12345))
    absent = fmix64_inverse((part << np.uint64(53)) | (np.arange(512, dtype=np.uint64) << np.uint64(44)) | np.uint64(999))
    return crafted, keys, absent, 0


def full_table(rng):
    """2,048 keys that look like some 600 to the estimate, one for each slot of the table that it asks for, and one of
    them so often that the pairs are not grouped by partitions."""
    keys = np.empty(2048, np.int64)
    absent = np.empty(2048, np.int64)
    for i in range(2048):
        h = (np.uint64(i) << np.uint64(53)) | rng.integers(0, 1 << 53, size=200, dtype=np.uint64)
        k = fmix64_inverse(h)
        low = k[(fmix64(k, 0x2545F4914F6CDD1D) >> np.uint64(53)) < np.uint64(512)]  # a quarter of the registers
        keys[i], absent[i] = low[0], low[1]
    return keys, np.empty(0, np.int64), absent, (1 << 20) - 5000


@pytest.mark.gpu
@pytest.mark.parametrize("make", [full_region, full_table])
def test_made_to_fill_the_table(make):
    import b2co
    import torch
    rng = np.random.default_rng(11)
    crafted, others, absent, heavy = make(rng)
    n = (1 << 20) + 3
    keys = np.concatenate([crafted, others])
    assert len(np.unique(keys)) == len(keys) and -1 not in keys and -1 not in absent
    once = np.arange(len(keys))
    fill = n - len(keys) - heavy
    # further pairs go to the other keys, or evenly over all
    more = rng.integers(len(crafted), len(keys), size=fill) if len(others) else rng.integers(0, len(keys), size=fill)
    at = rng.permutation(np.concatenate([once, np.full(heavy, 5), more]))
    v = rng.integers(-2**62, 2**62, size=n, dtype=np.int64)
    v[v == -1] = 0
    m = b2co.StaticMultimap(n, -1, -1, key_dtype=torch.int64, value_dtype=torch.int64)
    assert m.Insert(b2co.pack_pairs(dev(keys[at]), dev(v))) == 0
    q = np.concatenate([absent, keys])
    flags = torch.full((len(q),), 9, dtype=torch.uint8, device="cuda")
    m.Contains(dev(q), flags)
    assert np.array_equal(flags.cpu().numpy(), (np.arange(len(q)) >= len(absent)).astype(np.uint8))
    assert m.Count(dev(absent)) == 0
    assert m.Count(dev(q)) == n
    ko, vo = (torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(2))
    assert m.Retrieve(dev(q), ko, vo, n) == n
    order = np.lexsort((v, at))
    assert np.array_equal(ko.cpu().numpy(), keys[at[order]])
    assert np.array_equal(vo.cpu().numpy(), v[order])
    first = torch.zeros(len(absent), dtype=torch.int64, device="cuda")
    m.Find(dev(absent), first)
    assert (first.cpu().numpy() == -1).all()
