"""A table's first synchronous Insert leaves a stream capture that is going on beside it alone, and calls side
by side, more of them than a table has counters for, each get their own counts."""
import ctypes as C
import threading

import numpy as np
import pytest

from helpers import dev, make_pairs, unique_keys

pytestmark = pytest.mark.gpu


def new_map(slots):
    import b2co
    import torch
    return b2co.StaticMap(slots, -1, -1, key_dtype=torch.int64, value_dtype=torch.int64)


def test_first_insert_beside_a_capture():
    """The stream that is captured is one that the legacy stream waits for, so nothing may touch that one meanwhile."""
    import torch
    rng = np.random.default_rng(2)
    keys = unique_keys(rng, 3000, 8)
    pairs = make_pairs(keys, keys)
    again = torch.cat([pairs, pairs[:100]])
    q = dev(keys)
    out = torch.zeros(len(keys), dtype=torch.uint8, device="cuda")
    warm, t = new_map(10000), new_map(10000)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert warm.Insert(pairs, stream=side) == 0  # loads the kernels
    warm.Contains(q, out, stream=side)
    out.zero_()
    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.12")
    blocking, graph, instance = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(blocking)) == 0
    assert rt.cudaStreamBeginCapture(blocking, 2) == 0  # relaxed: other streams may be waited for
    try:
        warm.ContainsAsync(q, out, stream=blocking.value)
        assert t.Insert(again, stream=side) == 100
        assert t.InsertOrAssign(again, stream=side, with_assigned=True) == (0, 3100)
    finally:
        ended = rt.cudaStreamEndCapture(blocking, C.byref(graph))
    assert ended == 0
    assert rt.cudaGraphInstantiate(C.byref(instance), graph, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphLaunch(instance, blocking) == 0
    assert rt.cudaStreamSynchronize(blocking) == 0
    assert bool((out == 1).all())
    rt.cudaGraphExecDestroy(instance)
    rt.cudaGraphDestroy(graph)
    rt.cudaStreamDestroy(blocking)


def test_calls_side_by_side_have_their_own_counts():
    import torch
    rng = np.random.default_rng(3)
    threads, n = 12, 20000
    keys = unique_keys(rng, threads * n, 8)
    t = new_map(2 * threads * n)
    parts = [make_pairs(keys[i * n:(i + 1) * n], keys[i * n:(i + 1) * n]) for i in range(threads)]
    torch.cuda.synchronize()
    gate = threading.Barrier(threads)
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        for rep in range(20):
            gate.wait()
            fresh = rep == 0
            a = t.Insert(parts[i][: n - i], stream=s)  # another number of pairs in every thread
            b = t.InsertOrAssign(parts[i][: n - 2 * i], stream=s, with_assigned=True)
            if a != (0 if fresh else n - i) or b != (0, n - 2 * i):
                bad.append((i, rep, a, b))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for x in ts:
        x.start()
    for x in ts:
        x.join()
    assert not bad, bad[:5]
    # the counters are zero again: one more call counts every key that is there
    assert t.Insert(make_pairs(keys, keys)) == threads * n - sum(range(threads))
