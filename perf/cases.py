"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public Python layer (`b2co`) the way a program calls it: containers are created and
filled beforehand, inputs and output buffers lie on the GPU (pinned host buffers for the host-buffer lookup), and
one pass makes the calls of one step of such a program.  Sizes follow the repository's own benchmark configurations
(a 2^28-slot map, a 2^21-slot map, a 2^30-bit Bloom filter, a 64 KiB sketch, 4,096 log-normal tables, served requests
of 1,000 to 1,000,000 keys), with odd counts where a program would not have round ones.

listed() names the cases; draw() gives more of the same ranges; prepare() makes the inputs of a case from a seed;
run() is one pass and returns its outputs; work() is what one pass cannot do without.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ops-collections_b200"))
import b2co  # noqa: E402

# Slot layouts: (key dtype, payload dtype or None for a set).
LAYOUTS = {
    "i64i64": (torch.int64, torch.int64),
    "i32i32": (torch.int32, torch.int32),
    "i32i64": (torch.int32, torch.int64),
    "i64i32": (torch.int64, torch.int32),
    "i64": (torch.int64, None),
    "i32": (torch.int32, None),
}

# Probing schemes in use: the reference's defaults for maps and sets, and the other hash families.
SCHEMES = {
    "double_xxh32": (b2co.PROBE_DOUBLE, b2co.HASH_XXH32),
    "linear_murmur3": (b2co.PROBE_LINEAR, b2co.HASH_MURMUR3_32),
    "double_xxh64": (b2co.PROBE_DOUBLE, b2co.HASH_XXH64),
    "double_fmix": (b2co.PROBE_DOUBLE, b2co.HASH_FMIX),
}


def listed():
    return [
        # Bulk lookup in a table far larger than the caches: StaticMap<int64,int64> of 2^28 slots, half full,
        # 2^27 queries of which half hit (the headline workload).
        dict(name="find_large", kind="find", layout="i64i64", scheme="double_xxh32", slots=1 << 28, load=0.5,
             queries=1 << 27, hits=0.5, zipf=False),
        # The smallest request a server gets: 1,000 keys against a resident table; latency and launches count.
        dict(name="find_1k", kind="find", layout="i64i64", scheme="double_xxh32", slots=16666667, load=0.6,
             queries=1000, hits=0.7, zipf=False),
        # An ordinary served step: a small upsert and a lookup of 65,537 keys on a table of 50 M pairs, 70% hits.
        dict(name="request_64k", kind="upsert_find", layout="i64i64", scheme="double_xxh32", slots=83333333, load=0.6,
             queries=65537, updates=7001, hits=0.7),
        # A lookup table that fits the caches, built and asked within one step: 2^21 slots, 1 M int32 pairs.
        dict(name="small_map", kind="build_probe", layout="i32i32", scheme="double_xxh32", slots=1 << 21,
             pairs=1000000, queries=1000000, hits=0.5, contains=True),
        # A hash join: build on 40 M rows, probe with 60 M.
        dict(name="join", kind="build_probe", layout="i64i64", scheme="double_xxh32", slots=66666667, pairs=40000003,
             queries=60000011, hits=0.5, contains=False),
        # Deduplication / group-by: the first of equal keys wins, one input in ten repeats another.
        dict(name="dedup", kind="dedup", layout="i64i64", scheme="double_xxh32", slots=40000003, inputs=20000003,
             repeats=0.1),
        # Lookup for a program whose keys and results live in host memory.
        dict(name="find_host", kind="find_host", layout="i64i64", scheme="double_xxh32", slots=1 << 26, load=0.5,
             queries=(1 << 22) + 4097, hits=0.5),
        # A Bloom filter of 2^30 bits filled with 2^27 keys and asked for as many, half of them absent.
        dict(name="bloom", kind="bloom", key_bytes=8, blocks=1 << 22, adds=(1 << 27) + 11, queries=1 << 27, hits=0.5),
        # Counting distinct keys of a long stream: a 64 KiB sketch, 10^7 distinct int64 keys with repeats.
        dict(name="hll", kind="hll", key_bytes=8, precision=16, adds=(1 << 28) + 5, distinct=10000000),
        # Per-partition builds and probes: 4,096 int32 tables with log-normal key counts around 32,768.
        dict(name="group", kind="group", layout="i32i32", scheme="double_xxh32", tables=4096, median=32768),
        # A map that grew from 2^20 slots over eight batches: updates of present keys, then lookups.
        dict(name="dynamic", kind="dynamic", layout="i64i64", scheme="linear_murmur3", initial=1 << 20, batch=1 << 22,
             batches=8, updates=1 << 20, queries=(1 << 24) + 3, hits=0.5),
        # A join with repeated build keys: 2^24 pairs over 2^22 keys, counted and retrieved.
        dict(name="multimap", kind="multimap", layout="i64i64", entries=(1 << 24) + 1, distinct=1 << 22,
             queries=(1 << 21) + 7, hits=0.5),
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["find", "find", "upsert_find", "build_probe", "build_probe", "dedup", "find_host", "bloom",
                       "hll", "group", "dynamic", "multimap"])
    scheme = rng.choice(sorted(SCHEMES))
    maps = ["i64i64", "i32i32", "i32i64", "i64i32"]
    if kind == "find":
        slots = _log(rng, 1 << 14, 1 << 28)
        return dict(kind=kind, layout=rng.choice(sorted(LAYOUTS)), scheme=scheme, slots=slots,
                    load=rng.choice([0.3, 0.5, 0.6, 0.8]), queries=_log(rng, 500, 1 << 26),
                    hits=rng.choice([0.1, 0.5, 0.7, 1.0]), zipf=rng.random() < 0.25)
    if kind == "upsert_find":
        slots = _log(rng, 1 << 20, 1 << 27)
        queries = _log(rng, 1000, 1000000)
        return dict(kind=kind, layout=rng.choice(maps), scheme=scheme, slots=slots, load=0.6, queries=queries,
                    updates=min(queries // 9 + 1, slots // 4), hits=0.7)
    if kind == "build_probe":
        pairs = _log(rng, 10000, 40000000)
        return dict(kind=kind, layout=rng.choice(maps), scheme=scheme, slots=int(pairs / rng.choice([0.4, 0.5, 0.7])),
                    pairs=pairs, queries=int(pairs * rng.uniform(0.5, 1.5)), hits=rng.choice([0.2, 0.5, 1.0]),
                    contains=rng.random() < 0.5)
    if kind == "dedup":
        inputs = _log(rng, 20000, 20000000)
        return dict(kind=kind, layout=rng.choice(maps), scheme=scheme, slots=inputs * 2 + 1, inputs=inputs,
                    repeats=rng.choice([0.02, 0.1, 0.4]))
    if kind == "find_host":
        return dict(kind=kind, layout=rng.choice(["i64i64", "i32i32"]), scheme=scheme, slots=_log(rng, 1 << 20, 1 << 26),
                    load=0.5, queries=_log(rng, 20000, 4000000), hits=0.5)
    if kind == "bloom":
        blocks = _log(rng, 1 << 10, 1 << 22)
        return dict(kind=kind, key_bytes=rng.choice([4, 8]), blocks=blocks, adds=int(blocks * rng.uniform(1.0, 24.0)),
                    queries=int(blocks * rng.uniform(1.0, 24.0)), hits=rng.choice([0.1, 0.5, 0.9]))
    if kind == "hll":
        adds = _log(rng, 10000, 1 << 28)
        return dict(kind=kind, key_bytes=rng.choice([4, 8]), precision=rng.choice([13, 14, 16, 17]), adds=adds,
                    distinct=max(1000, int(adds * rng.uniform(0.02, 1.0))))
    if kind == "group":
        return dict(kind=kind, layout=rng.choice(["i32i32", "i64i64"]), scheme=scheme, tables=_log(rng, 32, 1024),
                    median=_log(rng, 2000, 60000))
    if kind == "dynamic":
        batch = _log(rng, 100000, 1 << 22)
        return dict(kind=kind, layout=rng.choice(["i64i64", "i32i32"]), scheme=scheme, initial=1 << 18, batch=batch,
                    batches=rng.randint(2, 6), updates=batch // 5 + 1, queries=_log(rng, 50000, 1 << 24), hits=0.5)
    entries = _log(rng, 20000, 1 << 24)
    return dict(kind="multimap", layout=rng.choice(maps), entries=entries,
                distinct=max(1, entries // rng.randint(2, 12)), queries=entries // rng.randint(2, 10) + 1,
                hits=rng.choice([0.5, 1.0]))


# ---- inputs: keys are a seeded bijection of item numbers, so a key is unique and known to be present or absent


def _shift(x, s):
    return (x >> s) & ((1 << (64 - s)) - 1)  # logical shift of int64


def _mix64(ids, seed):
    x = ids + ((seed * 0x9E3779B1 + 12345) & 0xFFFFFFFFFF) * (1 << 22)
    x = x ^ _shift(x, 30)
    x *= 0xBF58476D1CE4E5B9 - (1 << 64)
    x = x ^ _shift(x, 27)
    x *= 0x94D049BB133111EB - (1 << 64)
    return x ^ _shift(x, 31)


def _mix31(ids, seed):
    m = (1 << 31) - 1
    x = (ids * 0x2C1B3C6D + ((seed * 0x9E3779B1 + 977) & m)) & m
    x = x ^ (x >> 15)
    x = (x * 0x297A2D39) & m
    return x ^ (x >> 13)


def _keys(ids, dtype, seed):
    """Distinct keys of distinct item numbers: uniform int64, or uniform in [0, 2^31) for int32."""
    if dtype == torch.int64:
        return _mix64(ids, seed)
    return _mix31(ids, seed).to(torch.int32)


def _values(ids, dtype, seed):
    """Payloads that no sentinel meets."""
    v = _mix64(ids, seed + 7919)
    return (v & 0x7FFFFFFFFFFFFFF) if dtype == torch.int64 else (v & 0x7FFFFFFF).to(torch.int32)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _arange(n, start=0):
    return torch.arange(start, start + n, dtype=torch.int64, device="cuda")


def _query_ids(n, queries, hits, g, zipf=False):
    """Item numbers of a query stream over n present items (0..n-1): `hits` of them present, the others not."""
    if zipf:  # ranks of a Zipf(1.1) law over the present items
        u = torch.rand(queries, dtype=torch.float64, device="cuda", generator=g)
        top = float(n) ** -0.1 - 1.0
        return ((1.0 + u * top) ** -10.0).to(torch.int64).clamp_(1, n) - 1
    return torch.randint(0, max(n, int(n / hits)), (queries,), device="cuda", generator=g)


def _table(case):
    kd, vd = LAYOUTS[case["layout"]]
    probing, hash_kind = SCHEMES[case["scheme"]]
    if vd is None:
        return b2co.StaticSet(case["slots"], -1, key_dtype=kd, probing=probing, hash_kind=hash_kind)
    return b2co.StaticMap(case["slots"], -1, -1, key_dtype=kd, value_dtype=vd, probing=probing, hash_kind=hash_kind)


def _pairs(ids, layout, seed):
    """Pair array of a map (a key array of a set)."""
    kd, vd = LAYOUTS[layout]
    k = _keys(ids, kd, seed)
    return k if vd is None else b2co.pack_pairs(k, _values(ids, vd, seed))


def _filled(case, seed):
    t = _table(case)
    n = int(case["slots"] * case["load"])
    step = 1 << 26
    for at in range(0, n, step):
        t.Insert(_pairs(_arange(min(step, n - at), at), case["layout"], seed))
    return t, n


class _DeviceBytes:
    """A container's own device memory, as torch can read it."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(owner, ptr, n, typestr):
    return torch.as_tensor(_DeviceBytes(owner, ptr, n, typestr), device="cuda")


def _out_dtype(layout):
    kd, vd = LAYOUTS[layout]
    return kd if vd is None else vd


def _group_counts(case):
    """Keys of each table: the partitioning of a job, the same for every batch of data."""
    r = np.random.default_rng(case["tables"] * 1000003 + case["median"])
    c = r.lognormal(mean=math.log(case["median"]), sigma=1.2, size=case["tables"])
    return np.clip(c, 1024, 4194304).astype(np.int64)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case)
    if kind in ("find", "upsert_find", "build_probe", "dedup", "find_host", "group", "dynamic", "multimap"):
        kd, vd = LAYOUTS[case["layout"]]
        od = _out_dtype(case["layout"])
    if kind in ("find", "upsert_find", "find_host"):
        s["table"], n = _filled(case, seed)
        ids = _query_ids(n, case["queries"], case["hits"], g, case.get("zipf", False))
        s["keys"] = _keys(ids, kd, seed)
        s["out"] = torch.empty(case["queries"], dtype=od, device="cuda")
        if kind == "upsert_find":
            first = int(torch.randint(0, n - case["updates"], (1,), generator=g, device="cuda"))
            ids = _arange(case["updates"], first)
            ids = ids[torch.randperm(case["updates"], device="cuda", generator=g)]
            s["updates_in"] = b2co.pack_pairs(_keys(ids, kd, seed), _values(ids, vd, seed + 1))
        if kind == "find_host":
            np_dtype = {torch.int64: np.int64, torch.int32: np.int32}
            s["host_keys"] = b2co.pinned(case["queries"], np_dtype[kd])
            s["host_keys"][:] = s["keys"].cpu().numpy()
            s["host_out"] = b2co.pinned(case["queries"], np_dtype[od])
            del s["keys"], s["out"]
    elif kind == "build_probe":
        n = case["pairs"]
        s["table"] = _table(case)
        s["pairs_in"] = _pairs(_arange(n), case["layout"], seed)
        s["keys"] = _keys(_query_ids(n, case["queries"], case["hits"], g), kd, seed)
        s["out"] = torch.empty(case["queries"], dtype=od, device="cuda")
        s["flags"] = torch.empty(case["queries"], dtype=torch.uint8, device="cuda") if case["contains"] else None
    elif kind == "dedup":
        n = case["inputs"]
        s["table"] = _table(case)
        ids = _arange(n)
        again = torch.rand(n, device="cuda", generator=g) < case["repeats"]
        ids = torch.where(again, torch.randint(0, n, (n,), device="cuda", generator=g), ids)
        s["pairs_in"] = b2co.pack_pairs(_keys(ids, kd, seed), _values(_arange(n), vd, seed))
        s["found"] = torch.empty(n, dtype=od, device="cuda")
        s["inserted"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    elif kind == "bloom":
        kd = torch.int64 if case["key_bytes"] == 8 else torch.int32
        s["filter"] = b2co.BloomFilter(case["blocks"], key_dtype=kd)
        s["keys"] = _keys(_arange(case["adds"]), kd, seed)
        s["queries_in"] = _keys(_query_ids(case["adds"], case["queries"], case["hits"], g), kd, seed)
        s["flags"] = torch.empty(case["queries"], dtype=torch.uint8, device="cuda")
        s["words"] = _view(s["filter"], s["filter"].Data(), case["blocks"] * 8, "<i4")
    elif kind == "hll":
        kd = torch.int64 if case["key_bytes"] == 8 else torch.int32
        s["sketch"] = b2co.HyperLogLog(case["precision"], key_dtype=kd)
        ids = torch.randint(0, case["distinct"], (case["adds"],), device="cuda", generator=g)
        s["keys"] = _keys(ids, kd, seed)
        s["registers"] = _view(s["sketch"], s["sketch"].Data(), 1 << case["precision"], "|u1")
    elif kind == "group":
        counts = _group_counts(case)
        probing, hash_kind = SCHEMES[case["scheme"]]
        s["tables"] = b2co.TableGroup(2 * counts, -1, -1, key_dtype=kd, value_dtype=vd, probing=probing,
                                      hash_kind=hash_kind)
        total = int(counts.sum())
        c = torch.from_numpy(counts).cuda()
        off = torch.zeros(case["tables"] + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(c, 0, out=off[1:])
        s["pairs_in"] = _pairs(_arange(total), case["layout"], seed)
        s["pair_offsets"], s["key_offsets"] = off, off * 2
        # table t is asked 2 * counts[t] keys, each equally likely one of its own or an absent one
        table_of = torch.repeat_interleave(torch.arange(case["tables"], device="cuda"), 2 * c, output_size=2 * total)
        cq, oq = c[table_of], off[table_of]
        del table_of
        j = (torch.rand(2 * total, dtype=torch.float64, device="cuda", generator=g) * (2 * cq)).to(torch.int64)
        ids = torch.where(j < cq, oq + j, total + oq + (j - cq))
        del cq, oq, j
        s["keys"] = _keys(ids, kd, seed)
        s["out"] = torch.empty(2 * total, dtype=vd, device="cuda")
    elif kind == "dynamic":
        probing, hash_kind = SCHEMES[case["scheme"]]
        m = b2co.DynamicMap(case["initial"], -1, -1, -2, key_dtype=kd, value_dtype=vd, probing=probing,
                            hash_kind=hash_kind)
        n = case["batch"] * case["batches"]
        for b in range(case["batches"]):
            m.Insert(_pairs(_arange(case["batch"], b * case["batch"]), case["layout"], seed))
        ids = torch.randperm(n, device="cuda", generator=g)[: case["updates"]]
        up = b2co.pack_pairs(_keys(ids, kd, seed), _values(ids, vd, seed + 1))
        m.InsertOrAssign(up)  # the map has grown to the room that updates ask for
        s["map"], s["updates_in"] = m, up
        s["keys"] = _keys(_query_ids(n, case["queries"], case["hits"], g), kd, seed)
        s["out"] = torch.empty(case["queries"], dtype=vd, device="cuda")
        s["flags"] = torch.empty(case["queries"], dtype=torch.uint8, device="cuda")
    elif kind == "multimap":
        n, d = case["entries"], case["distinct"]
        s["map"] = b2co.StaticMultimap(n, -1, -1, key_dtype=kd, value_dtype=vd)
        ids = torch.randint(0, d, (n,), device="cuda", generator=g)
        s["pairs_in"] = b2co.pack_pairs(_keys(ids, kd, seed), _values(_arange(n), vd, seed))
        q = torch.randint(0, int(d / case["hits"]), (case["queries"],), device="cuda", generator=g)
        s["keys"] = _keys(q, kd, seed)
        room = int(1.5 * case["queries"] * case["hits"] * n / d) + 4096  # what a program sets aside for its matches
        s["key_out"] = torch.zeros(room, dtype=kd, device="cuda")
        s["value_out"] = torch.zeros(room, dtype=vd, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "find":
        if s["layout"] in ("i64", "i32"):  # a set is asked for membership as a rule
            s["table"].Contains(s["keys"], s["out"].view(torch.uint8))
            return s["out"].view(torch.uint8)[: s["queries"]]
        s["table"].Find(s["keys"], s["out"])
        return s["out"]
    if kind == "upsert_find":
        failed, assigned = s["table"].InsertOrAssign(s["updates_in"], with_assigned=True)
        s["table"].Find(s["keys"], s["out"])
        return {"failed": failed, "assigned": assigned, "out": s["out"]}
    if kind == "build_probe":
        t = s["table"]
        t.ClearAsync()
        failed = t.Insert(s["pairs_in"])
        t.Find(s["keys"], s["out"])
        if s["flags"] is not None:
            t.Contains(s["keys"], s["flags"])
        return {"failed": failed, "out": s["out"], "flags": s["flags"]}
    if kind == "dedup":
        t = s["table"]
        t.ClearAsync()
        t.InsertAndFind(s["pairs_in"], s["found"], s["inserted"], mode=b2co.IAF_FIRST_WINS)
        return {"found": s["found"], "inserted": s["inserted"]}
    if kind == "find_host":
        s["table"].FindHost(s["host_keys"], s["host_out"])
        return s["host_out"]
    if kind == "bloom":
        f = s["filter"]
        f.ClearAsync()
        f.Add(s["keys"])
        f.Contains(s["queries_in"], s["flags"])
        return {"words": s["words"], "flags": s["flags"]}
    if kind == "hll":
        h = s["sketch"]
        h.Clear()
        h.Add(s["keys"])
        return {"estimate": h.Estimate(), "registers": s["registers"]}
    if kind == "group":
        t = s["tables"]
        t.Clear()
        failed = t.Insert(s["pairs_in"], s["pair_offsets"])
        t.Find(s["keys"], s["key_offsets"], s["out"])
        return {"failed": failed, "out": s["out"]}
    if kind == "dynamic":
        m = s["map"]
        new = m.InsertOrAssign(s["updates_in"])
        m.Find(s["keys"], s["out"])
        m.Contains(s["keys"], s["flags"])
        return {"new": new, "size": m.Size(), "out": s["out"], "flags": s["flags"]}
    m = s["map"]
    m.Clear()
    failed = m.Insert(s["pairs_in"])
    total = m.Count(s["keys"])
    written = m.Retrieve(s["keys"], s["key_out"], s["value_out"], s["key_out"].shape[0])
    return {"failed": failed, "total": total, "written": written, "keys": s["key_out"], "values": s["value_out"]}


def _sizes(layout):
    kd, vd = LAYOUTS[layout]
    kb = torch.empty((), dtype=kd).element_size()
    vb = 0 if vd is None else torch.empty((), dtype=vd).element_size()
    return kb, vb, b2co.slot_bytes(kb, vb)


def work(case):
    """Bytes a pass cannot do without: inputs and outputs once, and of a table either one 32-byte sector per access
    or the whole table, whichever is less (a cleared table is written once)."""
    kind = case["kind"]
    if kind in ("find", "upsert_find", "find_host"):
        kb, vb, sb = _sizes(case["layout"])
        q, u = case["queries"], case.get("updates", 0)
        out = vb or 1
        touched = min(32 * q, case["slots"] * sb)
        return {"bytes": q * (kb + out) + touched + u * (sb + 64), "flops": 0}
    if kind == "build_probe":
        kb, vb, sb = _sizes(case["layout"])
        table = case["slots"] * sb
        q = case["queries"]
        flags = q * (kb + 1) if case["contains"] else 0
        return {"bytes": case["pairs"] * sb + table + min(32 * q, table) + q * (kb + vb) + flags, "flops": 0}
    if kind == "dedup":
        kb, vb, sb = _sizes(case["layout"])
        return {"bytes": case["inputs"] * (sb + vb + 1) + case["slots"] * sb, "flops": 0}
    if kind == "bloom":
        f = case["blocks"] * 32
        q = case["queries"]
        return {"bytes": case["adds"] * case["key_bytes"] + 2 * f + q * (case["key_bytes"] + 1), "flops": 0}
    if kind == "hll":
        return {"bytes": case["adds"] * case["key_bytes"] + 2 * (1 << case["precision"]), "flops": 0}
    if kind == "group":
        kb, vb, sb = _sizes(case["layout"])
        n = case["tables"] * case["median"] * math.exp(0.72)  # mean of the log-normal key count, sigma 1.2
        return {"bytes": n * sb + 2 * (2 * n * sb) + 2 * n * (kb + vb), "flops": 0}
    if kind == "dynamic":
        kb, vb, sb = _sizes(case["layout"])
        q, u = case["queries"], case["updates"]
        table = case["batch"] * case["batches"] * sb / 0.6
        return {"bytes": q * (2 * kb + vb + 1) + 2 * min(32 * q, table) + u * (sb + 64), "flops": 0}
    kb, vb, sb = _sizes(case["layout"])
    n, q = case["entries"], case["queries"]
    matches = q * case["hits"] * n / case["distinct"]
    return {"bytes": 2 * n * sb + 2 * q * kb + matches * (kb + 2 * vb), "flops": 0}
