"""The no-allocation build on two-byte slots, at the loads where its buckets
are the largest (32768 quotients, up to 24,000 items)."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodup", [True, False])
@pytest.mark.parametrize("load", [0.3, 0.6, 0.65, 0.7, 0.74])
@pytest.mark.parametrize("q", [15, 16, 18])
def test_noalloc_two_byte_slots(gqf, cuda, q, load, nodup):
    r = 13
    keys = O.mt_keys(800 + q, int(load * (1 << q)))
    t = O.sqf_new(q, r)
    assert O.sqf_bulk_build(t, q, r, keys, nodup) == 0
    f = gqf.initFilterGPU(q, r)
    try:
        d = to_dev(cuda, keys)
        cuda.cuda.synchronize()
        st = gqf.lib().gqf_sqf_bulk_build_noalloc(C.byref(f), keys.size, d.data_ptr(), int(nodup), None)
        assert st == gqf.GQF_OK
        assert np.array_equal(gqf.table_bytes(f), t)
    finally:
        gqf.freeFilterGPU(f)
