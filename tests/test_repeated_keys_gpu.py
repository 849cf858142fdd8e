"""Batches that repeat one fingerprint thousands of times: every occurrence
takes one stored copy, at a cost that does not grow with the square of the
copies."""
import numpy as np
import pytest

import oracle as O
from conftest import to_dev
from sqf_model import Contents, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sync", [True, False])
@pytest.mark.parametrize("q,r,copies", [(14, 5, 40), (16, 5, 2000), (18, 5, 30000), (16, 13, 700), (17, 13, 20000)])
def test_deletes_of_many_copies(gqf, cuda, q, r, copies, sync):
    keys = np.concatenate([np.full(copies, 99, np.uint32), O.mt_keys(900 + q, int(0.4 * (1 << q)))])
    near = keys[copies: copies + 500]
    c = Contents(q, r, keys, False)
    f = gqf.initFilterGPU(q, r)
    try:
        gqf.bulkBuildSegmentedLayouts(f, keys.size, to_dev(cuda, keys), False)
        part = np.concatenate([np.full(copies // 3, 99, np.uint32), near])
        for op, ref, k in ((gqf.superclusterDeletes, c.delete, part),
                           (gqf.insert, c.insert, part),  # all stored already but the deleted ones
                           (gqf.superclusterDeletes, c.delete, np.full(copies, 99, np.uint32))):
            op(f, k.size, to_dev(cuda, k), sync=sync)
            gqf.stream_status()
            ref(k)
            check(gqf, f, c.table(), op.__name__)
    finally:
        gqf.freeFilterGPU(f)


def test_deletes_of_30000_copies_are_not_quadratic(gqf, cuda):
    """A claim per copy already claimed made 4.5e8 atomics, 208 ms.  What is
    left is the rebuild's sort of one quotient's 60,000 items by one thread:
    about a million steps, 45 ms at the 13 ms that 20,000 items took."""
    q, r, copies = 20, 5, 30000
    keys = np.concatenate([np.full(copies, 99, np.uint32), O.mt_keys(950, 1 << 19)])
    f = gqf.initFilterGPU(q, r)
    try:
        dk, dd = to_dev(cuda, keys), to_dev(cuda, keys[:copies])
        ms = []
        for _ in range(2):
            gqf.bulkBuildSegmentedLayouts(f, keys.size, dk, False)
            ms.append(gqf.superclusterDeletes(f, copies, dd, sync=True))
        assert min(ms) < 120.0
    finally:
        gqf.freeFilterGPU(f)
