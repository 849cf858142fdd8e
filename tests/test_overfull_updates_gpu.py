"""Updates of filters with more fingerprints than quotients: clusters too long
to walk, and spills that pass whole buckets of the rebuild behind them."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


def distinct_keys(seed, q, r, n):
    k = O.mt_keys(seed, n + n // 4)
    u = k[np.sort(np.unique(O.aphash(k, q, r), return_index=True)[1])]
    assert u.size >= n
    return u[:n]


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("load", [1.03, 1.05])
@pytest.mark.parametrize("q,r", [(18, 5), (20, 5), (22, 5), (18, 13)])
def test_overfull_updates(gqf, cuda, q, r, load, sync):
    n, m = int(load * (1 << q)), 24
    keys = distinct_keys(850 + q, q, r, n + m)
    t = O.sqf_new(q, r)
    assert O.sqf_bulk_build(t, q, r, keys[:n], True) == 0
    f = gqf.initFilterGPU(q, r)
    try:
        gqf.bulkBuildSegmentedLayouts(f, n, to_dev(cuda, keys[:n]), True)
        assert np.array_equal(gqf.table_bytes(f), t)
        for op, ref, k in ((gqf.superclusterDeletes, O.sqf_delete, keys[:1]),
                           (gqf.insert, O.sqf_insert, keys[n:]),
                           (gqf.superclusterDeletes, O.sqf_delete, keys[n // 2: n // 2 + m])):
            op(f, k.size, to_dev(cuda, k), sync=sync)
            gqf.stream_status()
            ref(t, q, r, k)
            raw = gqf.table_bytes(f)
            assert np.array_equal(raw, t), "%s: %d bytes differ" % (op.__name__, np.count_nonzero(raw != t))
    finally:
        gqf.freeFilterGPU(f)
