"""Builds that keep every copy, and builds on two-byte slots: groups of one,
few and many items per quotient, buckets far over their average, nearly full
tables, queued and synchronous; the table byte for byte against the oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


def build_and_check(G, torch, q, r, keys, nodup):
    t = O.sqf_new(q, r)
    full = O.sqf_bulk_build(t, q, r, keys, nodup) != 0
    f = G.initFilterGPU(q, r)
    try:
        if full:  # too many for the slots past the last quotient: both say so
            with pytest.raises(G.GQFError) as e:
                G.bulkBuildSegmentedLayouts(f, keys.size, to_dev(torch, keys), nodup)
            assert e.value.status == G.GQF_ERR_FULL
            return
        for sync in (True, False):
            G.bulkBuildSegmentedLayouts(f, keys.size, to_dev(torch, keys), nodup, sync=sync)
            G.stream_status()
            raw = G.table_bytes(f)
            if not np.array_equal(raw, t):
                d = np.nonzero(raw != t)[0]
                raise AssertionError("sync=%s: %d bytes differ, first at %d" % (sync, d.size, d[0]))
    finally:
        G.freeFilterGPU(f)


@pytest.mark.parametrize("q,r,nodup", [(7, 5, False), (8, 13, True), (11, 13, False), (13, 5, False), (14, 13, True),
                                       (17, 5, False), (18, 13, True), (21, 5, False)])
@pytest.mark.parametrize("alpha", [0.01, 0.7, 1.04])
def test_group_build(gqf, cuda, q, r, nodup, alpha):
    build_and_check(gqf, cuda, q, r, O.mt_keys(700 + q, max(1, int(alpha * (1 << q)))), nodup)


@pytest.mark.parametrize("q,r,nodup", [(14, 5, False), (16, 13, True), (16, 13, False)])
def test_group_build_many_copies(gqf, cuda, q, r, nodup):
    """One key thousands of times, some tens of times, the rest once, and a
    narrow quotient range: groups past the sorted size, buckets past the
    shared memory they were sized for."""
    n = int(0.4 * (1 << q))
    few = O.mt_keys(720 + q, 40)
    cand = O.mt_keys(721, 1 << 20)
    narrow = cand[(O.aphash(cand, q, r) >> r) < 700][:600]
    keys = np.concatenate([np.full(5000, 99, np.uint32), np.repeat(few, 60), narrow, O.mt_keys(722 + q, n)])
    keys = keys[np.random.default_rng(1).permutation(keys.size)]
    build_and_check(gqf, cuda, q, r, keys, nodup)


@pytest.mark.parametrize("q,r,nodup", [(8, 5, False), (12, 13, True), (13, 13, False), (16, 5, False), (18, 13, True),
                                       (20, 5, False)])
@pytest.mark.parametrize("na,nb", [(0.45, 0.45), (0.7, 0.02), (0.0, 0.3)])
def test_group_merge(gqf, cuda, q, r, nodup, na, nb):
    """Merges that keep every copy, or of two-byte slots: both contents, one
    of them small, the first filter empty; one key a thousand times on both
    sides where the filter has room for it."""
    G, torch = gqf, cuda
    many = np.full(1000 if q >= 14 else 3, 99, np.uint32)
    a, b = O.mt_keys(740 + q, int(na * (1 << q))), np.concatenate([many, O.mt_keys(760 + q, int(nb * (1 << q)))])
    if na:
        a = np.concatenate([a, many])
    ta, tb = O.sqf_new(q, r), O.sqf_new(q, r)
    if na:
        assert O.sqf_bulk_build(ta, q, r, a, False) == 0
    assert O.sqf_bulk_build(tb, q, r, b, False) == 0
    assert O.sqf_merge_two(ta, tb.copy(), q, r, nodup) == 0
    for sync in (True, False):
        fa, fb = G.initFilterGPU(q, r), G.initFilterGPU(q, r)
        try:
            if na:
                G.bulkBuildSegmentedLayouts(fa, a.size, to_dev(torch, a), False)
            G.bulkBuildSegmentedLayouts(fb, b.size, to_dev(torch, b), False)
            G.mergeTwoFilters(fa, fb, nodup, sync=sync)
            G.stream_status()
            assert np.array_equal(G.table_bytes(fa), ta)
            assert np.array_equal(G.table_bytes(fb), tb)  # the second filter is only read
        finally:
            G.freeFilterGPU(fa)
            G.freeFilterGPU(fb)
