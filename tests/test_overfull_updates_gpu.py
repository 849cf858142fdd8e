"""Updates of filters with more fingerprints than quotients: clusters too long
to walk, and spills that pass whole buckets of the rebuild behind them."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev
from sqf_model import Contents, check

pytestmark = pytest.mark.gpu


def distinct_keys(seed, q, r, n):
    k = O.mt_keys(seed, n + n // 4)
    u = k[np.sort(np.unique(O.aphash(k, q, r), return_index=True)[1])]
    assert u.size >= n
    return u[:n]


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q,r,load", [(18, 5, 1.03), (18, 5, 1.05), (20, 5, 1.03), (20, 5, 1.05), (22, 5, 1.05),
                                      (18, 13, 1.03), (18, 13, 1.05)])
def test_overfull_updates(gqf, cuda, q, r, load, sync):
    n, m = int(load * (1 << q)), 24
    keys = distinct_keys(850 + q, q, r, n + m)
    c = Contents(q, r, keys[:n], True)
    f = gqf.initFilterGPU(q, r)
    try:
        gqf.bulkBuildSegmentedLayouts(f, n, to_dev(cuda, keys[:n]), True)
        check(gqf, f, c.table(), "build")
        for op, ref, k in ((gqf.superclusterDeletes, c.delete, keys[:1]), (gqf.insert, c.insert, keys[n:]),
                           (gqf.superclusterDeletes, c.delete, keys[n // 2: n // 2 + m])):
            op(f, k.size, to_dev(cuda, k), sync=sync)
            gqf.stream_status()
            ref(k)
            check(gqf, f, c.table(), op.__name__)
    finally:
        gqf.freeFilterGPU(f)
