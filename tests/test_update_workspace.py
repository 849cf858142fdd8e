"""gqf_sqf_update_workspace_bytes covers what every update of up to n keys
requests, on each of its routes: a reserved workspace does not grow."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from conftest import to_dev


def reported(G, q, r, n):
    return int(G.lib().gqf_sqf_update_workspace_bytes(q, r, n))


@pytest.mark.parametrize("q,r", [(7, 5), (15, 5), (18, 13), (20, 5), (22, 5), (24, 5), (26, 5)])
def test_reported_bytes_hold_the_buffers(gqf, q, r):
    """What an update cannot do without: an in-place one the table's snapshot,
    its contents as two lists of words and the batch's fingerprints, a
    cluster-local delete 24 bytes a key, an insert 24 with its hash set."""
    slots, table = O.sqf_num_slots(q), O.sqf_table_bytes(q, r)
    last = 0
    for n in sorted((0, 1, 1000, 1 << (q - 6), 1 << (q - 4), 1 << q, 1 << 22)):
        got = reported(gqf, q, r, n)
        assert got >= last  # smaller batches fit, too
        last = got
        assert got >= 8 * slots + 4 * n + (table if r == 5 else 0)
        if r == 13:
            assert got >= 24 * n
        elif q >= 22:
            assert got >= 24 * min(n, 1 << (q - 6))


@pytest.mark.gpu
@pytest.mark.parametrize("q,r,n", [(12, 5, 1 << 16), (16, 5, 1 << 20), (18, 13, 1 << 18), (20, 5, 1 << 20),
                                   (22, 5, 1 << 22), (23, 5, 1 << 17)])
def test_reserved_workspace_does_not_grow(gqf, cuda, q, r, n):
    G, L = gqf, gqf.lib()
    s = cuda.cuda.Stream()
    size = C.c_size_t()

    def held():
        assert L.gqf_workspace_reserve(C.c_void_p(s.cuda_stream), 0, C.byref(size)) == G.GQF_OK
        return size.value

    f = G.initFilterGPU(q, r)
    try:
        keys = to_dev(cuda, O.mt_keys(1200 + q, max(n, 1 << (q - 1))))
        G.bulkBuildSegmentedLayouts(f, 1 << (q - 1), keys, True)
        cuda.cuda.synchronize()
        assert L.gqf_workspace_reserve(C.c_void_p(s.cuda_stream), reported(G, q, r, n), C.byref(size)) == G.GQF_OK
        have = held()
        assert have >= reported(G, q, r, n)
        few = min(n, 1 << (q - 5))
        for sync in (True, False):
            for m in {n, 1 << (q - 6), 1 << (q - 4), 100}:
                if m > n:
                    continue
                G.superclusterDeletes(f, m, keys, stream=s, sync=sync)
                G.insert(f, min(m, few), keys, stream=s, sync=sync)
                assert held() == have, (m, sync)
        G.stream_status(s)
    finally:
        s.synchronize()
        G.freeFilterGPU(f)
        L.gqf_workspace_release(C.c_void_p(s.cuda_stream))
